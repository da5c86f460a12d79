// Energy equation: the implicit step of EnergyDirectSolve
// (SOURCE/ThermalRoutines.c:72-551) on the centroids, matrix-free.
//
// The reference assembles a five-point matrix (row per active centroid:
// rho Cv / dt plus the conductances k / h^2 of its faces, Dirichlet walls
// doubling the face conductance, the off-diagonals minus the conductances)
// and factorises it with CHOLMOD.  Here the same rows are applied on the fly
// (the diagonal and the right-hand side formed once per solve, exactly as the
// reference sums them) and the system, symmetric positive definite for the
// Cartesian case, is solved by conjugate gradients with the diagonal as
// preconditioner, in FP64, from the old temperature, in one launch that keeps
// the rows in shared memory where they fit.  Every inner product is
// a deterministic grid sum (fixed order), so a solve takes the same
// iterations and gives the same bits on every run.
#include <cmath>
#include "mdz_internal.cuh"

mdz_status mdz_ensure_fields(mdz_ctx *ctx);
mdz_status mdz_upload_fields(mdz_ctx *ctx, const mdz_fields *h, cudaStream_t st);
mdz_status mdz_download_fields(mdz_ctx *ctx, const mdz_fields *h, const char *const *names, int n, cudaStream_t st);

#define ZEROC_K 273.15

namespace {

constexpr int EN_THREADS = 256;
constexpr int EN_MAX_BLOCKS = 2048;   // partial slots per reduced value

struct energy_bc_dev {
    const signed char *type, *typW, *typE, *typS, *typN;
    const double *valW, *valE, *valS, *valN;
    double ixx, izz;   // 1/dx/dx, 1/dz/dz as the reference forms them (host: no FP64 division per row)
};

__device__ __forceinline__ bool active(const energy_bc_dev &B, int c) { return B.type[c] != 30; }

// Diagonal and right-hand side (b + bbc) of centroid row c, in the
// reference's order of additions (:158-187, :196-330).
__global__ void k_energy_setup(mdz_dgrid g, mdz_fields f, energy_bc_dev B, double dt, double gz, int shear,
                               int adiab, double *__restrict__ diag, double *__restrict__ rhs) {
    const int ncx = g.ncx, ncz = g.ncz, nx = g.Nx, nxvz = g.Nx + 1;
    const int c2 = blockIdx.x * blockDim.x + threadIdx.x;
    if (c2 >= ncx * ncz) return;
    const int k = c2 % ncx, l = c2 / ncx;
    if (!active(B, c2)) { diag[c2] = 1.0; rhs[c2] = 0.0; return; }
    const double ixx = B.ixx, izz = B.izz;
    const double rhoCp = f.rho_n[c2] * f.Cv[c2], T = f.T[c2];
    double b = 1.0 * rhoCp * T / dt;
    b += 1.0 * f.Qr[c2];
    if (shear == 1) b += f.Wdiss[c2];
    if (adiab == 1) {
        const int c3 = k + l * nxvz;
        b += T * f.alp[c2] * 0.5 * (f.v[c3 + 1] + f.v[c3 + 1 + nxvz]) * gz * f.rho_n[c2];
    } else if (adiab == 2) {
        b += T * f.alp[c2] * (f.p[c2] - f.p0_n[c2]) / dt;
    }
    const int c1 = k + (l + 1) * nx, c3 = k + l * nxvz + 1;
    const double AW = f.kx[c1], AE = f.kx[c1 + 1], AS = f.kz[c3], AN = f.kz[c3 + nxvz];
    double val = 1.0 * rhoCp / dt, bbc = 0.0;
    if (l > 0 && active(B, c2 - ncx)) val += AS * izz;
    if (k > 0 && active(B, c2 - 1)) val += AW * ixx;
    if (k < ncx - 1 && active(B, c2 + 1)) val += AE * ixx;
    if (l < ncz - 1 && active(B, c2 + ncx)) val += AN * izz;
    if (l == 0 && B.typS[k] == 1) { val += 2.0 * AS * izz; bbc += 2.0 * AS * izz * B.valS[k]; }
    if (l == 0 && B.typS[k] == 2) bbc += -1.0 / g.dx * B.valS[k];
    if (k == 0 && B.typW[l] == 1) { val += 2.0 * AW * ixx; bbc += 2.0 * AW * ixx * B.valW[l]; }
    if (k == ncx - 1 && B.typE[l] == 1) { val += 2.0 * AE * ixx; bbc += 2.0 * AE * ixx * B.valE[l]; }
    if (l == ncz - 1 && B.typN[k] == 1) { val += 2.0 * AN * izz; bbc += 2.0 * AN * izz * B.valN[k]; }
    diag[c2] = val;
    rhs[c2] = b + 1.0 * bbc;
}

// y = A x on the active rows (0 elsewhere); optionally dot = x . y over them
__device__ __forceinline__ double energy_row(const mdz_dgrid &g, const mdz_fields &f, const energy_bc_dev &B,
                                             const double *diag, const double *x, int c2) {
    const int ncx = g.ncx, ncz = g.ncz, nx = g.Nx, nxvz = g.Nx + 1;
    const int k = c2 % ncx, l = c2 / ncx;
    const double ixx = B.ixx, izz = B.izz;
    const int c1 = k + (l + 1) * nx, c3 = k + l * nxvz + 1;
    double y = diag[c2] * x[c2];
    if (l > 0 && active(B, c2 - ncx)) y += -1.0 * f.kz[c3] * izz * x[c2 - ncx];
    if (k > 0 && active(B, c2 - 1)) y += -1.0 * f.kx[c1] * ixx * x[c2 - 1];
    if (k < ncx - 1 && active(B, c2 + 1)) y += -1.0 * f.kx[c1 + 1] * ixx * x[c2 + 1];
    if (l < ncz - 1 && active(B, c2 + ncx)) y += -1.0 * f.kz[c3 + nxvz] * izz * x[c2 + ncx];
    return y;
}

// r = b - A x, z = r / diag, p = z; sums: r.z, r.r, b.b
__global__ void k_energy_init(mdz_dgrid g, mdz_fields f, energy_bc_dev B, const double *__restrict__ diag,
                              const double *__restrict__ rhs, const double *__restrict__ x, double *__restrict__ r,
                              double *__restrict__ z, double *__restrict__ p, double *part, unsigned int *cnt,
                              double *out) {
    double acc[3] = {0, 0, 0};
    const int n = g.ncx * g.ncz;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        double rr = 0.0, zz = 0.0;
        if (active(B, c)) {
            rr = rhs[c] - energy_row(g, f, B, diag, x, c);
            zz = rr / diag[c];
            acc[0] += rr * zz; acc[1] += rr * rr; acc[2] += rhs[c] * rhs[c];
        }
        r[c] = rr; z[c] = zz; p[c] = zz;
    }
    mdz_grid_sum<3, double>(acc, part, cnt, out);
}

// q = A p; sum p.q
__global__ void k_energy_apply(mdz_dgrid g, mdz_fields f, energy_bc_dev B, const double *__restrict__ diag,
                               const double *__restrict__ p, double *__restrict__ q, double *part, unsigned int *cnt,
                               double *out) {
    double acc[1] = {0};
    const int n = g.ncx * g.ncz;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        double y = 0.0;
        if (active(B, c)) {
            y = energy_row(g, f, B, diag, p, c);
            acc[0] += p[c] * y;
        }
        q[c] = y;
    }
    mdz_grid_sum<1, double>(acc, part, cnt, out);
}

// x += alpha p, r -= alpha q, z = r / diag; sums r.z, r.r   (alpha = s[0] / s[1])
__global__ void k_energy_update(int n, const signed char *__restrict__ type, const double *__restrict__ diag,
                                const double *__restrict__ s, const double *__restrict__ pq,
                                const double *__restrict__ p, const double *__restrict__ q, double *__restrict__ x,
                                double *__restrict__ r, double *__restrict__ z, double *part, unsigned int *cnt,
                                double *out) {
    const double alpha = s[0] / pq[0];
    double acc[2] = {0, 0};
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        if (type[c] == 30) continue;
        x[c] += alpha * p[c];
        const double rr = r[c] - alpha * q[c], zz = rr / diag[c];
        r[c] = rr;
        z[c] = zz;
        acc[0] += rr * zz;
        acc[1] += rr * rr;
    }
    mdz_grid_sum<2, double>(acc, part, cnt, out);
}

// p = z + beta p   (beta = s_new[0] / s_old[0])
__global__ void k_energy_dir(int n, const double *__restrict__ s_new, const double *__restrict__ s_old,
                             const double *__restrict__ z, double *__restrict__ p) {
    const double beta = s_new[0] / s_old[0];
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) p[c] = z[c] + beta * p[c];
}

// The whole of the conjugate gradients in one launch, for grids whose rows fit
// the chip's shared memory: CTA b owns the `m` consecutive cells from b m and
// keeps their diagonal, its reciprocal, the west and south couplings (east and
// north are the neighbours' own: the matrix is symmetric), r, q and p, the
// latter with the ncx cells before and after (their p is formed here too, from
// the z the neighbours wrote).  All CTAs are resident (cooperative launch, one
// per SM) and meet twice per iteration, at the two inner products.
//
// One launch per step of the recurrence (k_energy_apply, _update, _dir) costs
// three launches, two copies and a host wait per iteration, and the FP64 pipe,
// which bounds the sweeps (33 warps of cells per SM at 400 x 400, 16 clocks
// per warp instruction), spends its time on the conductance products and on
// the division by the diagonal, about 30 instructions per cell.  Held in
// shared memory as couplings and reciprocals a row takes 12.
//
// A meeting point is a 16-byte slot per CTA and value, {partial sum, epoch},
// written and read in one access each, so that arriving, waiting and fetching
// the partial sums are one trip through L2.  Slots of a kind are written again
// only after the other kind's meeting, that is after all have read them.
// Sums run over the slots in order: the same bits on every run.
constexpr int CG_THREADS = 512;
constexpr int CG_MAX_CTAS = CG_THREADS / 2;   // one CTA per SM; two values polled by a thread per slot
constexpr int CG_COPIES = 4;               // of every slot, so that 38 CTAs poll a line and not 152 (2.62 -> 2.44 ms at 400 x 400)
constexpr int CG_MIN_CELLS = 512;          // per CTA: below, a meeting costs more than the cells it spreads
constexpr unsigned CG_SPINS = 1u << 22;    // polls of a slot (some 2 s) before the solve is given up
constexpr int CG_RED = 2 * CG_THREADS + 32;   // partial sums of threads, of warps on arriving and of warps on collecting

struct alignas(16) cg_slot { unsigned long long sum, epoch; };

__device__ __forceinline__ void cg_post(cg_slot *s, double v, unsigned epoch) {
    asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.release.gpu.global.b128 [%0], t; }" ::"l"(s),
                 "l"(__double_as_longlong(v)), "l"((unsigned long long)epoch)
                 : "memory");
}

// Sums of NV values over the CTAs, in slot order, on thread 0 (and 256 for the
// second value).  Every slot has a thread of its own: with one warp polling
// five slots a lane one after the other the solve takes 2.98 ms, 2.62 so.
// False (on all threads): a CTA did not arrive.
template <int NV>
__device__ __forceinline__ bool cg_collect(const cg_slot *slot, unsigned epoch, double *red, double &sum) {
    const int t = threadIdx.x, i = t & (CG_MAX_CTAS - 1), G = gridDim.x;
    double v = 0.0;
    bool ok = true;
    if (t < NV * CG_MAX_CTAS && (i & ~31) < G) {
        if (i < G) {
            const cg_slot *s = slot + (t / CG_MAX_CTAS * CG_COPIES + blockIdx.x % CG_COPIES) * G + i;
            unsigned long long b, e;
            unsigned spin = 0;
            do {
                asm volatile("{ .reg .b128 t; ld.acquire.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
                             : "=&l"(b), "=&l"(e)
                             : "l"(s)
                             : "memory");
            } while (e != epoch && ++spin < CG_SPINS);
            ok = e == epoch;
            v = __longlong_as_double((long long)b);
        }
        __syncwarp();
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    }
    double *part = red + 2 * CG_THREADS + 16;
    if ((t & 31) == 0) part[t >> 5] = v;
    ok = __syncthreads_and(ok);
    if (i == 0 && t < NV * CG_MAX_CTAS) {
        const double *a = part + (t >> 5);
        sum = ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]));
    }
    return ok;
}

// Sums of NV values over the CTA, posted to the slots of this CTA: four warps
// per value fold the 512 partial sums to 128 and shuffle (35 warp
// instructions on the FP64 pipe; shuffles by all 16 warps take 85).
template <int NV>
__device__ __forceinline__ void cg_arrive(const double *acc, double *red, cg_slot *slot, unsigned epoch) {
    const int t = threadIdx.x;
    for (int v = 0; v < NV; v++) red[(v & 1) * CG_THREADS + t] = acc[v];
    __syncthreads();
    if (t < 128 * NV) {
        const double *a = red + (t >> 7) * CG_THREADS + (t & 127);
        double s = (a[0] + a[128]) + (a[256] + a[384]);
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if ((t & 31) == 0) red[2 * CG_THREADS + (t >> 5)] = s;
    }
    __syncthreads();
#pragma unroll
    for (int v = 0; v < NV; v++) {
        const unsigned copy = t - 128 * v;
        if (copy < CG_COPIES) {
            const double *a = red + 2 * CG_THREADS + 4 * v;
            cg_post(slot + (v * CG_COPIES + copy) * gridDim.x + blockIdx.x, (a[0] + a[1]) + (a[2] + a[3]), epoch);
        }
    }
}

struct cg_args {
    const double *diag, *rhs, *T;
    double *x, *z;
    cg_slot *slots;      // p.q, r.z, r.r, b.b: CG_COPIES x gridDim.x each
    double *rel;         // out
    int *its, *status;   // out; status 1: not finite, 2: a CTA did not arrive
    int n, m, max_its;
    double tol;
};

__global__ void __launch_bounds__(CG_THREADS, 1)
k_energy_cg(mdz_dgrid g, mdz_fields f, energy_bc_dev B, cg_args A) {
    extern __shared__ double sm[];
    __shared__ double s_num, s_rel, s_bnorm, s_stop;
    __shared__ int s_go;   // 1: on, 0: done, -1: not finite
    const int t = threadIdx.x, ncx = g.ncx, m = A.m, n = A.n, G = gridDim.x, c0 = blockIdx.x * m;
    const int own = min(m, n - c0);
    double *red = sm, *dg = red + CG_RED, *inv = dg + m, *r = inv + m, *q = r + m, *W = q + m, *S = W + m + 1;
    double *p = S + m + ncx + ncx;   // p[-ncx .. m + ncx)
    cg_slot *slot_q = A.slots, *slot_r = slot_q + CG_COPIES * G, *slot_b = slot_r + 2 * CG_COPIES * G;
    for (int i = t; i < m + ncx; i += CG_THREADS) {
        const int c = c0 + i;
        const bool in = c < n && active(B, c);
        const int k = c % ncx, l = c / ncx;
        if (i <= m) W[i] = in && k > 0 && active(B, c - 1) ? -1.0 * f.kx[k + (l + 1) * g.Nx] * B.ixx : 0.0;
        S[i] = in && l > 0 && active(B, c - ncx) ? -1.0 * f.kz[k + l * (g.Nx + 1) + 1] * B.izz : 0.0;
        if (i < m) {
            const double d = in ? A.diag[c] : 1.0;
            dg[i] = d;
            inv[i] = in ? 1.0 / d : 0.0;   // 0: r = z = p = 0 on inactive cells
        }
    }
    for (int i = t - ncx; i < m + ncx; i += CG_THREADS) {
        const int c = c0 + i;
        p[i] = c >= 0 && c < n && active(B, c) ? A.T[c] : 0.0;
    }
    __syncthreads();
    unsigned epoch = 1;
    {   // x = T, r = b - A x, z = r / diag
        double acc[2] = {0.0, 0.0}, bb[1] = {0.0};
        for (int i = t; i < own; i += CG_THREADS) {
            double rr = 0.0;
            if (active(B, c0 + i)) {
                const double b = A.rhs[c0 + i];
                rr = b - (dg[i] * p[i] + S[i] * p[i - ncx] + W[i] * p[i - 1] + W[i + 1] * p[i + 1] + S[i + ncx] * p[i + ncx]);
                bb[0] += b * b;
            }
            const double zz = rr * inv[i];
            A.x[c0 + i] = p[i];
            A.z[c0 + i] = q[i] = zz;
            r[i] = rr;
            acc[0] += rr * zz;
            acc[1] += rr * rr;
        }
        cg_arrive<1>(bb, red, slot_b, epoch);
        __syncthreads();
        cg_arrive<2>(acc, red, slot_r, epoch);
    }
    double num = 0.0;   // r.z, on thread 0
    bool first = true, ok = true;
    int it = 0, status = 0;
    for (;;) {
        // r.z on thread 0: beta; r.r (and b.b) on thread 256: the test on the residual.  1 / (old r.z)
        // is formed while the slots are on their way
        double s, b = 0.0;
        if (first) {
            ok = cg_collect<1>(slot_b, epoch, red, b);
            if (t == 0) {
                s_bnorm = sqrt(b);
                s_stop = b * A.tol * A.tol;
            }
            __syncthreads();
        }
        const double old = first || t ? 0.0 : 1.0 / num;
        ok = cg_collect<2>(slot_r, epoch, red, s) && ok;
        if (t == 0) {
            s_num = s * old;
            num = s;
        } else if (t == CG_MAX_CTAS) {
            // well above the tolerance: no root and no division on the way to the next iteration
            if (!first && it < A.max_its && s > 1.0001 * s_stop && s > 1e-280 && s < 1e300) {
                s_go = 1;
            } else {
                const double rel = s_bnorm > 0.0 ? sqrt(s) / s_bnorm : 0.0;
                s_rel = rel;
                s_go = !first && !isfinite(rel) ? -1 : rel > A.tol && it < A.max_its;
            }
        }
        __syncthreads();
        status = !ok ? 2 : s_go < 0 ? -s_go : 0;
        if (status || s_go == 0) break;
        const double beta = s_num;
        // p = z + beta p, the halo from the z that its owners wrote before the meeting
        for (int i = t - ncx; i < 0; i += CG_THREADS)
            if (c0 + i >= 0) p[i] = first ? __ldcg(A.z + c0 + i) : __ldcg(A.z + c0 + i) + beta * p[i];
        for (int i = m + t; i < m + ncx; i += CG_THREADS)
            if (c0 + i < n) p[i] = first ? __ldcg(A.z + c0 + i) : __ldcg(A.z + c0 + i) + beta * p[i];
        for (int i = t; i < own; i += CG_THREADS) p[i] = first ? q[i] : q[i] + beta * p[i];
        first = false;
        __syncthreads();
        // q = A p, p.q
        double pq[1] = {0.0};
        for (int i = t; i < own; i += CG_THREADS) {
            const double y =
                dg[i] * p[i] + S[i] * p[i - ncx] + W[i] * p[i - 1] + W[i + 1] * p[i + 1] + S[i + ncx] * p[i + ncx];
            q[i] = y;
            pq[0] += p[i] * y;
        }
        epoch++;
        cg_arrive<1>(pq, red, slot_q, epoch);
        ok = cg_collect<1>(slot_q, epoch, red, s);
        if (t == 0) s_num = num / s;
        __syncthreads();
        if (!ok) { status = 2; break; }
        const double alpha = s_num;
        // r -= alpha q, z = r / diag; x += alpha p while the sums are on their way
        double acc[2] = {0.0, 0.0};
        for (int i = t; i < own; i += CG_THREADS) {
            const double rr = r[i] - alpha * q[i], zz = rr * inv[i];
            r[i] = rr;
            A.z[c0 + i] = q[i] = zz;
            acc[0] += rr * zz;
            acc[1] += rr * rr;
        }
        epoch++;
        cg_arrive<2>(acc, red, slot_r, epoch);
        for (int i = t; i < own; i += CG_THREADS) A.x[c0 + i] += alpha * p[i];
        it++;
    }
    if (blockIdx.x == 0 && t == 0) {
        *A.its = it;
        *A.rel = s_rel;
        *A.status = status;
    }
}

// doubles of shared memory that k_energy_cg takes
size_t cg_doubles(int m, int ncx) { return CG_RED + 6 * (size_t)m + 1 + (size_t)m + 3 * (size_t)ncx; }

// T <- x, dT = x - T on active cells; air: dT = 0, T = 0 C; count T < 0
__global__ void k_energy_finish(int n, const signed char *__restrict__ type, const double *__restrict__ x,
                                double *__restrict__ T, double *__restrict__ dT, double t_air, int *neg) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    if (type[c] != 30) {
        dT[c] = 1.0 * (x[c] - T[c]);
        T[c] = T[c] + dT[c];
        if (T[c] < 0.0) atomicAdd(neg, 1);
    } else {
        dT[c] = 0.0;
        T[c] = t_air;
    }
}

}  // namespace

extern "C" mdz_status mdz_EnergyDirectSolve(mdz_ctx *ctx, mdz_fields *f, const mdz_thermal_bc *bc, double dt,
                                            double gz, int shear_heating, int adiab_heating, double scale_T,
                                            double rel_tol, int max_iterations, int *iterations,
                                            double *rel_residual) {
    if (!ctx || !f || !bc) return ctx ? mdz_fail(ctx, MDZ_ERR_ARG, "EnergyDirectSolve: null argument") : MDZ_ERR_ARG;
    if (!(dt > 0.0) || !(scale_T > 0.0))
        return mdz_fail(ctx, MDZ_ERR_ARG, "EnergyDirectSolve: dt and scale_T must be > 0");
    if (!bc->type || !bc->typW || !bc->typE || !bc->typS || !bc->typN || !bc->valW || !bc->valE || !bc->valS ||
        !bc->valN)
        return mdz_fail(ctx, MDZ_ERR_ARG, "EnergyDirectSolve: thermal boundary arrays missing");
    if (!f->T || !f->rho_n || !f->Cv || !f->Qr || !f->kx || !f->kz)
        return mdz_fail(ctx, MDZ_ERR_ARG, "EnergyDirectSolve: needs T, rho_n, Cv, Qr, kx, kz");
    if ((shear_heating == 1 && !f->Wdiss) || (adiab_heating == 1 && (!f->alp || !f->v)) ||
        (adiab_heating == 2 && (!f->alp || !f->p || !f->p0_n)))
        return mdz_fail(ctx, MDZ_ERR_ARG, "EnergyDirectSolve: heating terms need Wdiss / alp, v / alp, p, p0_n");
    const mdz_dgrid &g = ctx->g;
    const int ncx = g.ncx, ncz = g.ncz, n = ncx * ncz;
    for (int c = 0; c < n; c++)
        if (bc->type[c] != -1 && bc->type[c] != 30)
            return mdz_fail(ctx, MDZ_ERR_UNSUPPORTED,
                            "EnergyDirectSolve: centroid thermal tags other than -1 and 30 (free surface, periodic) "
                            "are not implemented");
    if (rel_tol <= 0.0) rel_tol = 1e-13;
    if (max_iterations <= 0) max_iterations = 10000;
    mdz_status s = mdz_ensure_fields(ctx);
    if (s != MDZ_OK) return s;
    cudaStream_t st = ctx->stream;
    if ((s = mdz_upload_fields(ctx, f, st)) != MDZ_OK) return s;
    // boundary arrays and work vectors in one staging buffer
    const size_t nb = (size_t)n + 2 * (ncx + ncz), nw = 2 * (size_t)(ncx + ncz);
    const size_t bytes = sizeof(double) * (7 * (size_t)n + nw + 8) + nb + 64 + 4 * CG_COPIES * sizeof(cg_slot) * CG_MAX_CTAS;
    unsigned char *buf = (unsigned char *)mdz_stage(ctx, 8, bytes);
    if (!buf) return mdz_fail(ctx, MDZ_ERR_CUDA, "EnergyDirectSolve: staging allocation failed");
    cg_slot *slots = (cg_slot *)buf;
    double *diag = (double *)(slots + 4 * CG_COPIES * CG_MAX_CTAS), *rhs = diag + n, *x = rhs + n, *r = x + n, *z = r + n, *p = z + n, *q = p + n;
    double *vals = q + n, *sc = vals + nw;   // sc: [0..2] init sums, [3] p.q, [4..5] update sums, [6] old r.z
    signed char *tags = (signed char *)(sc + 8);
    int *neg = (int *)(((uintptr_t)(tags + nb) + 15) & ~(uintptr_t)15);
    MDZ_CUDA(ctx, cudaMemcpyAsync(tags, bc->type, n, cudaMemcpyHostToDevice, st));
    MDZ_CUDA(ctx, cudaMemcpyAsync(tags + n, bc->typW, ncz, cudaMemcpyHostToDevice, st));
    MDZ_CUDA(ctx, cudaMemcpyAsync(tags + n + ncz, bc->typE, ncz, cudaMemcpyHostToDevice, st));
    MDZ_CUDA(ctx, cudaMemcpyAsync(tags + n + 2 * ncz, bc->typS, ncx, cudaMemcpyHostToDevice, st));
    MDZ_CUDA(ctx, cudaMemcpyAsync(tags + n + 2 * ncz + ncx, bc->typN, ncx, cudaMemcpyHostToDevice, st));
    MDZ_CUDA(ctx, cudaMemcpyAsync(vals, bc->valW, sizeof(double) * ncz, cudaMemcpyHostToDevice, st));
    MDZ_CUDA(ctx, cudaMemcpyAsync(vals + ncz, bc->valE, sizeof(double) * ncz, cudaMemcpyHostToDevice, st));
    MDZ_CUDA(ctx, cudaMemcpyAsync(vals + 2 * ncz, bc->valS, sizeof(double) * ncx, cudaMemcpyHostToDevice, st));
    MDZ_CUDA(ctx, cudaMemcpyAsync(vals + 2 * ncz + ncx, bc->valN, sizeof(double) * ncx, cudaMemcpyHostToDevice, st));
    MDZ_CUDA(ctx, cudaMemsetAsync(neg, 0, sizeof(int), st));
    energy_bc_dev B{tags, tags + n, tags + n + ncz, tags + n + 2 * ncz, tags + n + 2 * ncz + ncx,
                    vals, vals + ncz, vals + 2 * ncz, vals + 2 * ncz + ncx, 1.0 / g.dx / g.dx, 1.0 / g.dz / g.dz};
    const mdz_fields &d = ctx->d;
    k_energy_setup<<<mdz_blocks(n, EN_THREADS), EN_THREADS, 0, st>>>(g, d, B, dt, gz, shear_heating, adiab_heating,
                                                                      diag, rhs);
    MDZ_LAUNCHED(ctx);
    // One launch for the solve where the rows fit the SMs' shared memory (cg_doubles: on 152
    // SMs 539 904 cells at 1024 in a row, 559 000 in a square box): 2.4 ms the call at 400 x 400 (175 iterations; 10.2 by one launch per step of the
    // recurrence, three launches, two copies and a wait of the host per iteration), 1.6 at 200 x 100, 1.2 at
    // 59 x 32; beyond, the sweeps outweigh the launches
    int dev = 0, sms = 0, smem = 0, it = 0;
    double rel = 0.0;
    MDZ_CUDA(ctx, cudaGetDevice(&dev));
    MDZ_CUDA(ctx, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    MDZ_CUDA(ctx, cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    int G = (n + CG_MIN_CELLS - 1) / CG_MIN_CELLS;
    G = G < sms ? G : sms;
    G = G < CG_MAX_CTAS ? G : CG_MAX_CTAS;
    const int m = ((n + G - 1) / G + 31) / 32 * 32;
    G = (n + m - 1) / m;
    const size_t cg_bytes = sizeof(double) * cg_doubles(m, ncx);
    bool done = false;
    if (cg_bytes + 64 <= (size_t)smem) {
        // (the kernel's limit belongs to the process: the same value from every call, whatever its grid, so that no other
        // thread's call lowers it between here and the launch)
        MDZ_CUDA(ctx, cudaFuncSetAttribute(k_energy_cg, cudaFuncAttributeMaxDynamicSharedMemorySize, smem - 64));
        cg_args A{diag, rhs, d.T, x, z, slots, sc, neg + 1, neg + 2, n, m, max_iterations, rel_tol};
        MDZ_CUDA(ctx, cudaMemsetAsync(slots, 0, 4 * CG_COPIES * sizeof(cg_slot) * G, st));
        void *args[] = {(void *)&g, (void *)&d, (void *)&B, (void *)&A};
        const cudaError_t e =
            cudaLaunchCooperativeKernel((const void *)k_energy_cg, dim3(G), dim3(CG_THREADS), args, cg_bytes, st);
        // a device (or a part of one) that cannot hold the whole grid refuses the launch: the steps below need no such thing
        done = e != cudaErrorCooperativeLaunchTooLarge && e != cudaErrorLaunchOutOfResources && e != cudaErrorNotSupported;
        if (!done) (void)cudaGetLastError();
        else if (e != cudaSuccess) return mdz_cuda_check(ctx, e, "EnergyDirectSolve");
    }
    if (done) {
        MDZ_LAUNCHED(ctx);
        int out[2];
        MDZ_CUDA(ctx, cudaMemcpyAsync(&rel, sc, sizeof rel, cudaMemcpyDeviceToHost, st));
        MDZ_CUDA(ctx, cudaMemcpyAsync(out, neg + 1, sizeof out, cudaMemcpyDeviceToHost, st));
        MDZ_CUDA(ctx, cudaStreamSynchronize(st));
        it = out[0];
        if (out[1] == 1) return mdz_fail(ctx, MDZ_ERR_NAN, "EnergyDirectSolve: NaN residual");
        if (out[1]) return mdz_fail(ctx, MDZ_ERR_CUDA, "EnergyDirectSolve: the CTAs of the solve did not meet");
    } else {
        MDZ_CUDA(ctx, cudaMemcpyAsync(x, d.T, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));   // start: old T
        int blocks = mdz_blocks(n, EN_THREADS);
        if (blocks > EN_MAX_BLOCKS) blocks = EN_MAX_BLOCKS;
        double *part = ctx->red_part + MDZ_RP_ENERGY;
        unsigned int *cnt = ctx->red_cnt + MDZ_RC_ENERGY;
        k_energy_init<<<blocks, EN_THREADS, 0, st>>>(g, d, B, diag, rhs, x, r, z, p, part, cnt, sc);
        MDZ_LAUNCHED(ctx);
        double h[3];
        MDZ_CUDA(ctx, cudaMemcpyAsync(h, sc, sizeof h, cudaMemcpyDeviceToHost, st));
        MDZ_CUDA(ctx, cudaStreamSynchronize(st));
        const double bnorm = std::sqrt(h[2]);
        rel = bnorm > 0.0 ? std::sqrt(h[1]) / bnorm : 0.0;
        // sc[0]: r.z of the current iteration (the update kernel reads it as the
        // numerator of alpha), sc[4]: the new r.z; they swap roles through sc[6]
        while (rel > rel_tol && it < max_iterations) {
            k_energy_apply<<<blocks, EN_THREADS, 0, st>>>(g, d, B, diag, p, q, part + 0, cnt + 1, sc + 3);
            MDZ_LAUNCHED(ctx);
            k_energy_update<<<blocks, EN_THREADS, 0, st>>>(n, tags, diag, sc, sc + 3, p, q, x, r, z, part + 2048,
                                                            cnt + 2, sc + 4);
            MDZ_LAUNCHED(ctx);
            k_energy_dir<<<blocks, EN_THREADS, 0, st>>>(n, sc + 4, sc, z, p);
            MDZ_LAUNCHED(ctx);
            MDZ_CUDA(ctx, cudaMemcpyAsync(sc, sc + 4, sizeof(double), cudaMemcpyDeviceToDevice, st));
            double u[2];
            MDZ_CUDA(ctx, cudaMemcpyAsync(u, sc + 4, sizeof u, cudaMemcpyDeviceToHost, st));
            MDZ_CUDA(ctx, cudaStreamSynchronize(st));
            rel = bnorm > 0.0 ? std::sqrt(u[1]) / bnorm : 0.0;
            it++;
            if (!std::isfinite(rel)) return mdz_fail(ctx, MDZ_ERR_NAN, "EnergyDirectSolve: NaN residual");
        }
    }
    if (iterations) *iterations = it;
    if (rel_residual) *rel_residual = rel;
    k_energy_finish<<<mdz_blocks(n), MDZ_THREADS, 0, st>>>(n, tags, x, d.T, d.dT, ZEROC_K / scale_T, neg);
    MDZ_LAUNCHED(ctx);
    static const char *const names[] = {"T", "dT"};
    if ((s = mdz_download_fields(ctx, f, names, 2, st)) != MDZ_OK) return s;
    int nneg = 0;
    MDZ_CUDA(ctx, cudaMemcpyAsync(&nneg, neg, sizeof(int), cudaMemcpyDeviceToHost, st));
    MDZ_CUDA(ctx, cudaStreamSynchronize(st));
    if (rel > rel_tol)
        return mdz_fail(ctx, MDZ_ERR_NOT_CONVERGED, "EnergyDirectSolve: relative residual %.3e after %d iterations",
                        rel, it);
    if (nneg) return mdz_fail(ctx, MDZ_ERR_STATE, "EnergyDirectSolve: negative temperature in %d cells", nneg);
    return MDZ_OK;
}
