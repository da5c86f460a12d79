// V-cycle kernels that do two phases of a level in one launch, on tiles in
// shared memory:
//   residual + restriction   the fine residual of the rows a tile of coarse
//                            points reads goes to shared memory only, and the
//                            coarse right-hand side is written together with
//                            the coarse level's first sweep from x = 0
//                            (x = omega D^-1 f)
//   prolongation + sweep     x + P x_coarse of a tile and its halo in shared
//                            memory, then one damped Jacobi sweep from it
// A level of a V-cycle with 2 + 1 sweeps is three launches instead of six.
//
// Every kernel here is launched with programmatic dependent launch
// (launch_pdl): it fetches what no launch of the V-cycle writes (stencils,
// inverse diagonals) and only then waits for the launch before it.  On the
// small levels a launch is mostly latency (its own start, then one trip to L2
// for the stencil rows and one for the vectors); this way the first two
// overlap the launch before.
// FP32 kernels also release the next launch at once (mg_release).  FP64 kernels
// do not: their blocks are bound by the SM's few FP64 units, and blocks of the
// next launch that arrive early gather on the SMs that happen to be free.
// One V-cycle, 1025 x 513 in FP32: 131 us without programmatic launches, 130
// with them, 109 with the early release; 257 x 129 in FP64: 107, 105 and 159.
// (Before the fused phases: 205 and 218 us.)
#pragma once

template <typename T>
__device__ __forceinline__ void mg_release() {
    if constexpr (sizeof(T) == 4) pdl_release();
}

struct box_geom {
    int Nx, Nz, ncx, ncz;
};

// A transfer weight (0 or a normal float) in the level's precision, without
// the conversion instruction: FP64 instructions, conversions among them,
// issue at a small fraction of the FP32 rate on this part.
template <typename T>
__device__ __forceinline__ T weight(float w) {
    if constexpr (sizeof(T) == 8) {
        const int b = __float_as_int(w);
        return b == 0 ? T(0) : __hiloint2double((b >> 3) + 0x38000000, b << 29);
    } else {
        return w;
    }
}

// ---- transfers ---------------------------------------------------------------
// x + P xc at fine u node (k, l) / v node (i, j); 0 outside the box
template <typename T, typename GF, typename GC>
__device__ __forceinline__ T prolonged_u(const GF &F, const GC &Cg, const T *cu, const T *xu, int k, int l) {
    const int Nx = F.Nx, Nxc = Cg.Nx;
    if (k < 0 || k >= Nx || l < 0 || l > F.Nz) return T(0);
    T x = xu[k + l * Nx];
    if (u_unknown(k, l, Nx, F.Nz)) {   // Vx: x node-centred, z cell-centred
        int J0, J1;
        float w0, w1;
        cc_weights(l, Cg.ncz, J0, w0, J1, w1);
        const int Ia = k >> 1, Ib = (k + 1) >> 1;
        const float wa = (k & 1) ? 0.5f : 1.0f, wb = (k & 1) ? 0.5f : 0.0f;
        const T a0 = cu[Ia + J0 * Nxc], a1 = cu[Ia + J1 * Nxc], b0 = cu[Ib + J0 * Nxc], b1 = cu[Ib + J1 * Nxc];
        x += weight<T>(wa * w0) * a0 + weight<T>(wa * w1) * a1 + weight<T>(wb * w0) * b0 + weight<T>(wb * w1) * b1;
    }
    return x;
}

template <typename T, typename GF, typename GC>
__device__ __forceinline__ T prolonged_v(const GF &F, const GC &Cg, const T *cv, const T *xv, int i, int j) {
    const int Nx = F.Nx, W = Cg.Nx + 1;
    if (i < 0 || i > Nx || j < 0 || j >= F.Nz) return T(0);
    T x = xv[i + j * (Nx + 1)];
    if (v_unknown(i, j, Nx, F.Nz)) {   // Vz: x cell-centred, z node-centred
        int I0, I1;
        float w0, w1;
        cc_weights(i, Cg.ncx, I0, w0, I1, w1);
        const int Ja = j >> 1, Jb = (j + 1) >> 1;
        const float wa = (j & 1) ? 0.5f : 1.0f, wb = (j & 1) ? 0.5f : 0.0f;
        const T a0 = cv[I0 + Ja * W], a1 = cv[I1 + Ja * W], b0 = cv[I0 + Jb * W], b1 = cv[I1 + Jb * W];
        x += weight<T>(wa * w0) * a0 + weight<T>(wa * w1) * a1 + weight<T>(wb * w0) * b0 + weight<T>(wb * w1) * b1;
    }
    return x;
}

// fine x += P xc (a V-cycle without post-smoothing)
template <typename T>
__global__ void k_mg_prolong_add(stokes_geom F, stokes_geom Cg, const T *cu, const T *cv, T *fu, T *fv) {
    mg_release<T>();
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i < F.Nx && j <= F.Nz) fu[i + j * F.Nx] = prolonged_u<T>(F, Cg, cu, fu, i, j);
    if (i <= F.Nx && j < F.Nz) fv[i + j * (F.Nx + 1)] = prolonged_v<T>(F, Cg, cv, fv, i, j);
}

// Weight of fine line 2 J - 2 + a (a = 0..3, cell-centred direction) for
// coarse line J: 1/4, 3/4, 3/4, 1/4, and the lines next to the walls, whose
// ghost parents are mirrored, count in full.
__device__ __forceinline__ float cc_restrict_weight(int J, int a, int ncc) {
    if (a == 0 || a == 3) return 0.25f;
    return (a == 1 ? J == 1 : J == ncc) ? 1.0f : 0.75f;
}

// (P^T r)(I, J) of one component from a fine residual that is zero outside the unknowns
template <typename T, typename GF, typename GC>
__device__ __forceinline__ T restricted_u(const GF &F, const GC &Cg, const T *ru, int I, int J) {
    T s = 0;
#pragma unroll
    for (int a = 0; a < 4; a++) {
        const float wz = cc_restrict_weight(J, a, Cg.ncz);
        const T *p = ru + min(2 * J - 2 + a, F.Nz) * F.Nx + 2 * I - 1;
#pragma unroll
        for (int b = 0; b < 3; b++) s += weight<T>((b == 1 ? 1.0f : 0.5f) * wz) * p[b];
    }
    return s;
}

template <typename T, typename GF, typename GC>
__device__ __forceinline__ T restricted_v(const GF &F, const GC &Cg, const T *rv, int I, int J) {
    T s = 0;
#pragma unroll
    for (int a = 0; a < 4; a++) {
        const float wx = cc_restrict_weight(I, a, Cg.ncx);
        const T *p = rv + (2 * J - 1) * (F.Nx + 1) + min(2 * I - 2 + a, F.Nx);
#pragma unroll
        for (int b = 0; b < 3; b++) s += weight<T>(wx * (b == 1 ? 1.0f : 0.5f)) * p[b * (F.Nx + 1)];
    }
    return s;
}

// ---- stencil levels ---------------------------------------------------------
// out = x + omega D^-1 (f - A x) on a stencil level (x == nullptr: x = 0),
// one thread per row (u rows first, then v rows), small blocks so that the
// levels of a few thousand rows spread over the SMs
#define ST_THREADS 64
template <typename T>
__global__ void __launch_bounds__(ST_THREADS) k_st_smooth(
    stokes_geom G, const T *__restrict__ su, const T *__restrict__ sv, const T *xu, const T *xv, const T *fu,
    const T *fv, const T *__restrict__ idu, const T *__restrict__ idv, T omega, T *__restrict__ ou,
    T *__restrict__ ov) {
    mg_release<T>();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int Nx = G.Nx, Nz = G.Nz, nu = Nx * (Nz + 1), nv = (Nx + 1) * Nz;
    if (t >= nu + nv) return;
    T cf[MG_NST], r = 0;
    if (t < nu) {
        const int i = t % Nx, j = t / Nx;
        const bool unk = u_unknown(i, j, Nx, Nz);
        T d = 0;
        if (unk) {
            if (xu) st_coefs<T>(su, nu, t, cf);
            d = idu[t];
        }
        pdl_wait();
        if (unk) {
            if (xu) r = xu[t] + omega * d * (fu[t] - st_urow_x<T>(Nx, Nz, cf, xu, xv, i, j));
            else r = omega * d * fu[t];
        }
        ou[t] = r;
    } else {
        const int c = t - nu, i = c % (Nx + 1), j = c / (Nx + 1);
        const bool unk = v_unknown(i, j, Nx, Nz);
        T d = 0;
        if (unk) {
            if (xu) st_coefs<T>(sv, nv, c, cf);
            d = idv[c];
        }
        pdl_wait();
        if (unk) {
            if (xv) r = xv[c] + omega * d * (fv[c] - st_vrow_x<T>(Nx, Nz, cf, xu, xv, i, j));
            else r = omega * d * fv[c];
        }
        ov[c] = r;
    }
}

// Coarse tile TX x TY per block: (2 TX + 1) x (2 TY + 2) fine u rows and
// (2 TX + 2) x (2 TY + 1) fine v rows.
template <typename T, int TX, int TY>
__device__ __forceinline__ void restrict_tile(const stokes_geom &Cg,
                                              const T (&ru)[2 * TY + 2][2 * TX + 1],
                                              const T (&rv)[2 * TY + 1][2 * TX + 2], int I0, int J0,
                                              T *__restrict__ cu, T *__restrict__ cv, const T *__restrict__ cidu,
                                              const T *__restrict__ cidv, T omega, T *__restrict__ cxu,
                                              T *__restrict__ cxv) {
    const int Nx = Cg.Nx, Nz = Cg.Nz;
    for (int t = threadIdx.x; t < 2 * TX * TY; t += blockDim.x) {
        const int p = t % (TX * TY), li = p % TX, lj = p / TX, I = I0 + li, J = J0 + lj;
        if (t < TX * TY) {
            if (I >= Nx || J > Nz) continue;
            T s = 0, x0 = 0;
            const int c = I + J * Nx;
            if (u_unknown(I, J, Nx, Nz)) {
#pragma unroll
                for (int a = 0; a < 4; a++) {
                    const float wz = cc_restrict_weight(J, a, Cg.ncz);
#pragma unroll
                    for (int b = 0; b < 3; b++) s += weight<T>((b == 1 ? 1.0f : 0.5f) * wz) * ru[2 * lj + a][2 * li + b];
                }
                if (cxu) x0 = omega * cidu[c] * s;
            }
            cu[c] = s;
            if (cxu) cxu[c] = x0;
        } else {
            if (I > Nx || J >= Nz) continue;
            T s = 0, x0 = 0;
            const int c = I + J * (Nx + 1);
            if (v_unknown(I, J, Nx, Nz)) {
#pragma unroll
                for (int a = 0; a < 4; a++) {
                    const float wx = cc_restrict_weight(I, a, Cg.ncx);
#pragma unroll
                    for (int b = 0; b < 3; b++) s += weight<T>(wx * (b == 1 ? 1.0f : 0.5f)) * rv[2 * lj + b][2 * li + a];
                }
                if (cxv) x0 = omega * cidv[c] * s;
            }
            cv[c] = s;
            if (cxv) cxv[c] = x0;
        }
    }
}

template <typename T, int TX, int TY, int NT>
__global__ void __launch_bounds__(NT) k_st_resid_restrict(
    stokes_geom F, const T *__restrict__ su, const T *__restrict__ sv, const T *xu, const T *xv, const T *fu,
    const T *fv, stokes_geom Cg, T *__restrict__ cu, T *__restrict__ cv, const T *__restrict__ cidu,
    const T *__restrict__ cidv, T omega, T *__restrict__ cxu, T *__restrict__ cxv) {
    constexpr int UW = 2 * TX + 1, UH = 2 * TY + 2, VW = 2 * TX + 2, VH = 2 * TY + 1;
    __shared__ T ru[UH][UW], rv[VH][VW];
    const int Nx = F.Nx, Nz = F.Nz, I0 = blockIdx.x * TX, J0 = blockIdx.y * TY;
    const size_t nu = (size_t)Nx * (Nz + 1), nv = (size_t)(Nx + 1) * Nz;
    mg_release<T>();
    if (sizeof(T) == 8 && !cxu) pdl_release();   // the bottom kernel follows: 8 CTAs that load while this one runs
#pragma unroll 1
    for (int t0 = 0; t0 < UW * UH + VW * VH; t0 += NT) {
        const int t = t0 + threadIdx.x;
        const bool u = t < UW * UH;
        const int q = u ? t : t - UW * UH, w = u ? UW : VW, a = q % w, b = q / w;
        const int k = 2 * I0 - (u ? 1 : 2) + a, l = 2 * J0 - (u ? 2 : 1) + b;
        const bool row = t < UW * UH + VW * VH, unk = row && (u ? u_unknown(k, l, Nx, Nz) : v_unknown(k, l, Nx, Nz));
        const int c = u ? k + l * Nx : k + l * (Nx + 1);
        T cf[MG_NST], r = 0;
        if (unk) st_coefs<T>(u ? su : sv, u ? nu : nv, c, cf);
        if (t0 == 0) pdl_wait();
        if (unk) r = u ? fu[c] - st_urow_x<T>(Nx, Nz, cf, xu, xv, k, l) : fv[c] - st_vrow_x<T>(Nx, Nz, cf, xu, xv, k, l);
        if (!row) continue;
        if (u) ru[b][a] = r;
        else rv[b][a] = r;
    }
    __syncthreads();
    restrict_tile<T, TX, TY>(Cg, ru, rv, I0, J0, cu, cv, cidu, cidv, omega, cxu, cxv);
}

// Tile of TW x TH points, one thread per row (TW TH u rows, then as many v
// rows); each thread loads its row's coefficients before the tile is filled.
template <typename T, int TW, int TH>
__global__ void __launch_bounds__(2 * TW * TH) k_st_prolong_smooth(
    stokes_geom F, stokes_geom Cg, const T *__restrict__ su, const T *__restrict__ sv, const T *cu, const T *cv,
    const T *xu, const T *xv, const T *fu, const T *fv, const T *__restrict__ idu, const T *__restrict__ idv, T omega,
    T *__restrict__ ou, T *__restrict__ ov) {
    constexpr int PUW = TW + 3, PUH = TH + 4, PVW = TW + 4, PVH = TH + 3, NT = 2 * TW * TH;
    __shared__ T pu[PUH][PUW], pv[PVH][PVW];   // u from (i0 - 2, j0 - 2), v from (i0 - 2, j0 - 2)
    const int Nx = F.Nx, Nz = F.Nz, i0 = blockIdx.x * TW, j0 = blockIdx.y * TH;
    const bool urow = threadIdx.x < TW * TH;
    const int p = threadIdx.x % (TW * TH), li = p % TW, lj = p / TW, i = i0 + li, j = j0 + lj;
    const bool inside = urow ? (i < Nx && j <= Nz) : (i <= Nx && j < Nz);
    const bool unk = urow ? u_unknown(i, j, Nx, Nz) : v_unknown(i, j, Nx, Nz);
    const size_t c = urow ? (size_t)i + (size_t)j * Nx : (size_t)i + (size_t)j * (Nx + 1);
    const size_t n = urow ? (size_t)Nx * (Nz + 1) : (size_t)(Nx + 1) * Nz;
    mg_release<T>();
    T cf[MG_NST], f = 0, d = 0;
    if (unk) {
        st_coefs<T>(urow ? su : sv, n, c, cf);
        d = urow ? idu[c] : idv[c];
    }
    pdl_wait();
    if (unk) f = urow ? fu[c] : fv[c];
    for (int t = threadIdx.x; t < PUW * PUH + PVW * PVH; t += NT) {
        if (t < PUW * PUH) {
            const int a = t % PUW, b = t / PUW;
            pu[b][a] = prolonged_u<T>(F, Cg, cu, xu, i0 - 2 + a, j0 - 2 + b);
        } else {
            const int q = t - PUW * PUH, a = q % PVW, b = q / PVW;
            pv[b][a] = prolonged_v<T>(F, Cg, cv, xv, i0 - 2 + a, j0 - 2 + b);
        }
    }
    __syncthreads();
    if (!inside) return;
    T r = 0;
    if (unk) {
        constexpr int NA = sizeof(T) == 8 ? 4 : 1;   // as st_urow_x
        T a[NA] = {}, s;
        if (urow) {
#pragma unroll
            for (int q = 0; q < 15; q++) a[q % NA] += cf[q] * pu[lj + q / 3][li + 1 + q % 3];
#pragma unroll
            for (int q = 0; q < 16; q++) a[(15 + q) % NA] += cf[15 + q] * pv[lj + q / 4][li + 1 + q % 4];
            if constexpr (NA == 4) s = (a[0] + a[1]) + (a[2] + a[3]);
            else s = a[0];
            r = pu[lj + 2][li + 2] + omega * d * (f - s);
        } else {
#pragma unroll
            for (int q = 0; q < 15; q++) a[q % NA] += cf[q] * pv[lj + 1 + q / 5][li + q % 5];
#pragma unroll
            for (int q = 0; q < 16; q++) a[(15 + q) % NA] += cf[15 + q] * pu[lj + 1 + q / 4][li + q % 4];
            if constexpr (NA == 4) s = (a[0] + a[1]) + (a[2] + a[3]);
            else s = a[0];
            r = pv[lj + 2][li + 2] + omega * d * (f - s);
        }
    }
    if (urow) ou[c] = r;
    else ov[c] = r;
}

// ---- level 0 of a Picard hierarchy (viscosities read directly) ---------------
// Picard momentum rows of the free-slip box that every hierarchy starts from
// (checked before it is built; no tags are read).  A block first forms the
// stresses its rows difference, once per centroid and vertex, into shared
// memory, with the cell volume and the grid spacings folded into their
// constants:
//   sx = D11 (2/3 du/dx - 1/3 dw/dz) dz      sz = D11 (2/3 dw/dz - 1/3 du/dx) dx
//   g  = D33 (du/dz + dw/dx) dx              (0 on the walls: free slip)
//   A u = (sx_W - sx_E) + (g_S - g_N)        A w = (sz_S - sz_N) + (dz / dx) (g_W - g_E)
// In FP64 these kernels are bound by the FP64 pipe (80 % active): evaluated
// row by row (picard_urow / picard_vrow) a point cost 60 FP64 instructions, from
// the tile about 27; 401^2 sweep 24 -> 15 us, residual + restriction 34 -> 19,
// prolongation + sweep 29 -> 20.  FP32 has the instructions to spare and no use
// for the extra barrier (one V-cycle at 1025 x 513: 109 us row by row, 118 from
// the tile), so it evaluates row by row.
template <typename T>
constexpr bool mg_stress_tile() { return sizeof(T) == 8; }

// rates of an accessor X.u(k, l), X.v(k, l)
template <typename T, typename VEL>
struct rates_of {
    VEL X;
    T idx, idz;
    __device__ __forceinline__ pair2<T> exx(int kc, int lc) const {
        const T dudx = (X.u(kc + 1, lc + 1) - X.u(kc, lc + 1)) * idx, dvdz = (X.v(kc + 1, lc + 1) - X.v(kc + 1, lc)) * idz;
        const T div = dudx + dvdz;
        return pair2<T>{dudx - div * T(1.0 / 3.0), dvdz - div * T(1.0 / 3.0)};
    }
    __device__ __forceinline__ T gxz(int kv, int lv) const {
        return (X.u(kv, lv + 1) - X.u(kv, lv)) * idz + (X.v(kv + 1, lv) - X.v(kv, lv)) * idx;
    }
};
template <typename T, typename VEL>
__device__ __forceinline__ T picard_urow(const stokes_geom &G, const stokes_coefs<T> &D, int k, int l, const VEL &X) {
    const rates_of<T, VEL> rs{X, gc<T>(G, GC_IDX), gc<T>(G, GC_IDZ)};
    const int nx = G.Nx, c1 = k + l * nx, c2 = k - 1 + (l - 1) * G.ncx;
    const T TxxE = D.D11[c2 + 1] * rs.exx(k, l - 1).x, TxxW = D.D11[c2] * rs.exx(k - 1, l - 1).x;
    const T TxzN = l < G.Nz - 1 ? D.D33[c1] * rs.gxz(k, l) : T(0), TxzS = l > 1 ? D.D33[c1 - nx] * rs.gxz(k, l - 1) : T(0);
    return (-(TxxE - TxxW) * rs.idx - (TxzN - TxzS) * rs.idz) * gc<T>(G, GC_CELVOL);
}
template <typename T, typename VEL>
__device__ __forceinline__ T picard_vrow(const stokes_geom &G, const stokes_coefs<T> &D, int k, int l, const VEL &X) {
    const rates_of<T, VEL> rs{X, gc<T>(G, GC_IDX), gc<T>(G, GC_IDZ)};
    const int c1 = k + l * G.Nx, c2 = k - 1 + (l - 1) * G.ncx;
    const T TzzN = D.D22[c2 + G.ncx] * rs.exx(k - 1, l).y, TzzS = D.D22[c2] * rs.exx(k - 1, l - 1).y;
    const T TxzE = k < G.Nx - 1 ? D.D33[c1] * rs.gxz(k, l) : T(0), TxzW = k > 1 ? D.D33[c1 - 1] * rs.gxz(k - 1, l) : T(0);
    return (-(TzzN - TzzS) * rs.idz - (TxzE - TxzW) * rs.idx) * gc<T>(G, GC_CELVOL);
}

template <typename T, int W, int H>
struct visc_tile {
    T sx[H][W], sz[H][W], g[H][W];   // centroids and vertices from (x0, z0)
    // X: X.u(k, l), X.v(k, l) at nodes inside the box
    template <typename VEL>
    __device__ __forceinline__ void fill(const stokes_geom &G, const stokes_coefs<T> &D, const VEL &X, int x0, int z0,
                                         int tid, int nt) {
        const T dx = gc<T>(G, GC_DX), dz = gc<T>(G, GC_DZ), idx = gc<T>(G, GC_IDX), idz = gc<T>(G, GC_IDZ);
        const T third = T(1.0 / 3.0), xx = T(2) * third * (dz * idx), xz = third, zz = T(2) * third * (dx * idz),
                gx = dx * idz;
        for (int t = tid; t < W * H; t += nt) {
            const int a = t % W, b = t / W, k = x0 + a, l = z0 + b;
            T vx = 0, vz = 0, vg = 0;
            if (k >= 0 && k < G.ncx && l >= 0 && l < G.ncz) {
                const T du = X.u(k + 1, l + 1) - X.u(k, l + 1), dv = X.v(k + 1, l + 1) - X.v(k + 1, l);
                const T d = D.D11[k + l * G.ncx];
                vx = d * (xx * du - xz * dv);
                vz = d * (zz * dv - xz * du);
            }
            if (k >= 1 && k <= G.Nx - 2 && l >= 1 && l <= G.Nz - 2)
                vg = D.D33[k + l * G.Nx] * (gx * (X.u(k, l + 1) - X.u(k, l)) + (X.v(k + 1, l) - X.v(k, l)));
            sx[b][a] = vx;
            sz[b][a] = vz;
            g[b][a] = vg;
        }
    }
    // rows at point (k, l) = tile position (a, b): centroid (k - 1, l - 1) is (a - 1, b - 1)
    __device__ __forceinline__ T urow(int a, int b) const {
        return (sx[b - 1][a - 1] - sx[b - 1][a]) + (g[b - 1][a] - g[b][a]);
    }
    __device__ __forceinline__ T vrow(int a, int b, T ratio) const {
        return (sz[b - 1][a - 1] - sz[b][a - 1]) + ratio * (g[b][a - 1] - g[b][a]);
    }
};

template <typename T>
struct vel_global {
    const T *xu, *xv;
    int Nx;
    __device__ __forceinline__ T u(int k, int l) const { return xu[k + l * Nx]; }
    __device__ __forceinline__ T v(int i, int j) const { return xv[i + j * (Nx + 1)]; }
};

// out = x + omega * D^-1 (f - A x)  (x == nullptr: x = 0), TW x TH points per block
template <typename T, int TW, int TH>
__global__ void __launch_bounds__(TW *TH) k_mg_smooth(stokes_geom G, stokes_coefs<T> D, const T *xu, const T *xv,
                                                   const T *fu, const T *fv, const T *__restrict__ idu,
                                                   const T *__restrict__ idv, T omega, T *__restrict__ ou,
                                                   T *__restrict__ ov) {
    constexpr bool TILE = mg_stress_tile<T>();
    __shared__ visc_tile<T, TILE ? TW + 1 : 1, TILE ? TH + 1 : 1> S;
    mg_release<T>();
    pdl_wait();
    const int i0 = blockIdx.x * TW, j0 = blockIdx.y * TH, a = threadIdx.x % TW, b = threadIdx.x / TW;
    const int i = i0 + a, j = j0 + b, Nx = G.Nx, Nz = G.Nz;
    const vel_global<T> X{xu, xv, Nx};
    if (TILE && xu) {
        S.fill(G, D, X, i0 - 1, j0 - 1, threadIdx.x, TW * TH);
        __syncthreads();
    }
    const T ratio = gc<T>(G, GC_DZ) * gc<T>(G, GC_IDX);
    auto au = [&]() { if constexpr (TILE) return S.urow(a + 1, b + 1); else return picard_urow<T>(G, D, i, j, X); };
    auto av = [&]() { if constexpr (TILE) return S.vrow(a + 1, b + 1, ratio); else return picard_vrow<T>(G, D, i, j, X); };
    if (i < Nx && j <= Nz) {
        const int c = i + j * Nx;
        T r = 0;
        if (u_unknown(i, j, Nx, Nz)) r = xu ? xu[c] + omega * idu[c] * (fu[c] - au()) : omega * idu[c] * fu[c];
        ou[c] = r;
    }
    if (i <= Nx && j < Nz) {
        const int c = i + j * (Nx + 1);
        T r = 0;
        if (v_unknown(i, j, Nx, Nz)) r = xv ? xv[c] + omega * idv[c] * (fv[c] - av()) : omega * idv[c] * fv[c];
        ov[c] = r;
    }
}

template <typename T, int TX, int TY, int NT>
__global__ void __launch_bounds__(NT) k_mg_resid_restrict(stokes_geom F, stokes_coefs<T> D, const T *xu, const T *xv,
                                                          const T *fu, const T *fv, stokes_geom Cg,
                                                          T *__restrict__ cu, T *__restrict__ cv,
                                                          const T *__restrict__ cidu, const T *__restrict__ cidv,
                                                          T omega, T *__restrict__ cxu, T *__restrict__ cxv) {
    constexpr int UW = 2 * TX + 1, UH = 2 * TY + 2, VW = 2 * TX + 2, VH = 2 * TY + 1;
    __shared__ T ru[UH][UW], rv[VH][VW];
    constexpr bool TILE = mg_stress_tile<T>();
    __shared__ visc_tile<T, TILE ? 2 * TX + 3 : 1, TILE ? 2 * TY + 3 : 1> S;   // from (2 I0 - 3, 2 J0 - 3)
    const int Nx = F.Nx, Nz = F.Nz, I0 = blockIdx.x * TX, J0 = blockIdx.y * TY;
    mg_release<T>();
    if (sizeof(T) == 8 && !cxu) pdl_release();   // (as in k_st_resid_restrict)
    pdl_wait();
    const vel_global<T> X{xu, xv, Nx};
    if constexpr (TILE) {
        S.fill(F, D, X, 2 * I0 - 3, 2 * J0 - 3, threadIdx.x, NT);
        __syncthreads();
    }
    const T ratio = gc<T>(F, GC_DZ) * gc<T>(F, GC_IDX);
    for (int t = threadIdx.x; t < UW * UH + VW * VH; t += NT) {
        T r = 0;
        if (t < UW * UH) {
            const int a = t % UW, b = t / UW, k = 2 * I0 - 1 + a, l = 2 * J0 - 2 + b;
            if (u_unknown(k, l, Nx, Nz)) {
                if constexpr (TILE) r = fu[k + l * Nx] - S.urow(a + 2, b + 1);
                else r = fu[k + l * Nx] - picard_urow<T>(F, D, k, l, X);
            }
            ru[b][a] = r;
        } else {
            const int q = t - UW * UH, a = q % VW, b = q / VW, i = 2 * I0 - 2 + a, j = 2 * J0 - 1 + b;
            if (v_unknown(i, j, Nx, Nz)) {
                if constexpr (TILE) r = fv[i + j * (Nx + 1)] - S.vrow(a + 1, b + 2, ratio);
                else r = fv[i + j * (Nx + 1)] - picard_vrow<T>(F, D, i, j, X);
            }
            rv[b][a] = r;
        }
    }
    __syncthreads();
    restrict_tile<T, TX, TY>(Cg, ru, rv, I0, J0, cu, cv, cidu, cidv, omega, cxu, cxv);
}

// velocities of a tile in shared memory that starts at node (i0, j0) of both components
template <typename T, int W>
struct vel_tile {
    const T (*pu)[W], (*pv)[W];
    int i0, j0;
    __device__ __forceinline__ T u(int k, int l) const { return pu[l - j0][k - i0]; }
    __device__ __forceinline__ T v(int k, int l) const { return pv[l - j0][k - i0]; }
};

template <typename T, int TW, int TH>
__global__ void __launch_bounds__(TW *TH) k_mg_prolong_smooth(
    stokes_geom F, stokes_coefs<T> D, stokes_geom Cg, const T *cu, const T *cv, const T *xu, const T *xv, const T *fu,
    const T *fv, const T *__restrict__ idu, const T *__restrict__ idv, T omega, T *__restrict__ ou, T *__restrict__ ov,
    T *zp, const double *pmean) {
    constexpr int W = TW + 2, H = TH + 2;
    constexpr bool TILE = mg_stress_tile<T>();
    __shared__ T pu[H][W], pv[H][W];
    __shared__ visc_tile<T, TILE ? TW + 1 : 1, TILE ? TH + 1 : 1> S;
    mg_release<T>();
    pdl_wait();
    const int Nx = F.Nx, Nz = F.Nz, i0 = blockIdx.x * TW, j0 = blockIdx.y * TH;
    for (int t = threadIdx.x; t < W * H; t += TW * TH) {
        const int a = t % W, b = t / W;
        pu[b][a] = prolonged_u<T>(F, Cg, cu, xu, i0 - 1 + a, j0 - 1 + b);
        pv[b][a] = prolonged_v<T>(F, Cg, cv, xv, i0 - 1 + a, j0 - 1 + b);
    }
    __syncthreads();
    const vel_tile<T, W> X{pu, pv, i0 - 1, j0 - 1};
    if constexpr (TILE) {
        S.fill(F, D, X, i0 - 1, j0 - 1, threadIdx.x, TW * TH);
        __syncthreads();
    }
    const int a = threadIdx.x % TW, b = threadIdx.x / TW, i = i0 + a, j = j0 + b;
    const T ratio = gc<T>(F, GC_DZ) * gc<T>(F, GC_IDX);
    auto au = [&]() { if constexpr (TILE) return S.urow(a + 1, b + 1); else return picard_urow<T>(F, D, i, j, X); };
    auto av = [&]() { if constexpr (TILE) return S.vrow(a + 1, b + 1, ratio); else return picard_vrow<T>(F, D, i, j, X); };
    if (i < Nx && j <= Nz) {
        const int c = i + j * Nx;
        T r = 0;
        if (u_unknown(i, j, Nx, Nz)) r = pu[b + 1][a + 1] + omega * idu[c] * (fu[c] - au());
        ou[c] = r;
    }
    if (i <= Nx && j < Nz) {
        const int c = i + j * (Nx + 1);
        T r = 0;
        if (v_unknown(i, j, Nx, Nz)) r = pv[b + 1][a + 1] + omega * idv[c] * (fv[c] - av());
        ov[c] = r;
    }
    if (zp && i < F.ncx && j < F.ncz) zp[i + j * F.ncx] -= (T)pmean[2];   // as k_pmean_out
}
