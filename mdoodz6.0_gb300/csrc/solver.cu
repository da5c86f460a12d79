// Linear solver for the decoupled Stokes correction  K dx = F  (K = Picard
// operator or Newton Jacobian, applied matrix-free): right-preconditioned,
// restarted GCR with classical Gram-Schmidt and a selective second pass, FP64
// dot products (fixed-order block sums), and an upper block-triangular
// preconditioner [[A, B], [0, S]]:
//   S^-1 = eta_n / cell volume            (viscosity-scaled pressure mass)
//   A^-1 = one geometric-multigrid V-cycle on the velocity block (Picard,
//          or optionally the Newton Jacobian's): damped Jacobi smoothing,
//          cell counts halved (odd ones rounded up), bilinear prolongation, R = P^T,
//          Galerkin coarse operators R A P as 31-point stencils, and an
//          explicit inverse (or a single-CTA Jacobi-PCG solve) on the
//          coarsest level.
// The same code runs in FP64 (plain form) and with FP32 storage and FP32
// stencil / V-cycle arithmetic (T = float) inside an FP64 defect-correction
// loop (iterative refinement); all inner products accumulate in FP64.
//
// This replaces the reference's CHOLMOD-preconditioned GCR with
// Powell-Hestenes iterations (KillerSolver, SOURCE/Solvers.c:2226-2755 and
// kspgcr, SOURCE/Solvers.c:100-228): same defect-correction equation, solved to
// a relative tolerance, without assembling a matrix.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <atomic>
#include <thread>
#include <vector>
#include "stokes.cuh"
#include "solver.cuh"
#include "krylov_dots.cuh"

#define MG_MAX_LEVELS 16
#define MG_DENSE_MAX 256
#define MG_DENSE_SMEM (200 * 1024)  // the coarsest level is inverted in shared memory up to this size (FP64: n <= 160)
#define MG_NST 31        // stencil coefficients per velocity row (15 same-component + 16 cross)
#define MG_CENTER 7      // plane of the diagonal entry in both layouts
#define GCR_MAX_M 48
#define GCR_NOTE 32       // slots of mdz_solver::sc the device writes: running squared norm, ticket
#define MG_TILE_LARGE 30000   // points of a level above which the restriction takes the larger tile
#define MG_TILE_SMALL 4000    // and below which the tile kernels take the smallest

// ---------------------------------------------------------------------------
template <typename T>
struct mg_level {
    int Nx = 0, Nz = 0, ncx = 0, ncz = 0;
    double dx = 0, dz = 0;
    signed char *BCu = nullptr, *BCv = nullptr, *BCp = nullptr, *BCg = nullptr;
    bool own_tags = false;
    T *D11 = nullptr, *D33 = nullptr;           // level 0 (Picard): D11 = D22 = 2 eta_n; D33 = eta_s
    // 31-point stencils of the velocity block (MG_NST coefficient planes per
    // component, structure of arrays): level 0 probed from the re-discretised
    // operator, coarser levels the Galerkin product R A P of the level above.
    T *su = nullptr, *sv = nullptr;
    T *pz = nullptr;                            // level 0: zero pressure vector for Newton probes
    T *xu = nullptr, *xv = nullptr, *yu = nullptr, *yv = nullptr;
    T *fu = nullptr, *fv = nullptr, *ru = nullptr, *rv = nullptr;
    T *idu = nullptr, *idv = nullptr;
    T *cg[8] = {nullptr};                       // coarsest-level CG workspace
    // coarsest level with at most MG_DENSE_MAX unknowns: explicit inverse
    int ndense = 0;
    int *dmap = nullptr;                        // dense index -> u index, or nu + v index
    T *Awork = nullptr;                         // ndense^2: the elimination, where it does not fit in shared memory
    T *AinvT = nullptr;                         // inverse, column-major
    size_t nu() const { return (size_t)Nx * (Nz + 1); }
    size_t nv() const { return (size_t)(Nx + 1) * Nz; }
    stokes_geom geom() const { return make_geom(Nx, Nz, dx, dz, BCu, BCv, BCp, BCg); }
    stokes_coefs<T> coefs() const {
        return stokes_coefs<T>{D11, nullptr, nullptr, nullptr, nullptr, D11, nullptr, nullptr,
                               nullptr, nullptr, D33, nullptr};
    }
};

template <typename T>
struct gcr_space {
    size_t nu = 0, nv = 0, np = 0, n = 0;
    size_t ld = 0;                      // n rounded up to whole 128-byte lines: the vectors' stride and allocated
                                        // length, zero beyond n, so that the vector kernels load 16 bytes a thread
    int m = 0;
    T *Z = nullptr, *W = nullptr;       // m basis vectors each (u, v, p contiguous)
    T *x = nullptr, *r = nullptr, *z = nullptr, *w = nullptr, *t = nullptr;
    T *pin = nullptr;                   // the preconditioner's input (graph-captured pointer)
    double *tri = nullptr;              // Gram-Schmidt triangle U (column q at q * GCR_MAX_M), then gamma
    const T **dA0 = nullptr;            // table of the dot products' vectors
    double *dots = nullptr;             // device scalars
    // FP32 copies of the operator (only used for T = float)
    T *Dc[12] = {nullptr};
};

template <typename T>
struct mg_hier {
    int nlev = 0;
    bool newton = false;          // level 0 is the probed Newton block (smoothed by its stencil)
    bool built = false;           // mg_setup has filled the levels at least once
    bool viscous = false;         // the last mg_setup left level 0 to its viscosities (no stencils stored)
    bool bottom = false;          // the device can place k_mg_bottom's cluster
    stokes_geom setup_geom{};     // level 0 of that set-up
    double *pmean = nullptr;      // preconditioner scratch: pressure sum, count and mean
    mg_level<T> L[MG_MAX_LEVELS];
};

#define MDZ_PRE_SLOTS 8
struct mdz_solver {
    mg_hier<double> mg64;
    mg_hier<float> mg32;
    gcr_space<double> g64;
    gcr_space<float> g32;
    double *sc = nullptr;        // host-pinned scalars
    double ticket = 0.0;         // of the newest GCR iteration (gcr_wait_note)
    bool ready = false;
    int nu1 = 2, nu2 = 1;        // fewer sweeps, a few more Krylov iterations: faster overall at 1025x513
    double omega = 0.7;
    int check = 1;               // GCR iterations between host convergence checks (one read-back
                                 // each: cheaper at 1025x513 than the iterations a sparser check overshoots)
    int restart = 30;            // GCR basis size
    int mg_jacobian = 0;         // 1: multigrid on the Newton Jacobian's velocity block (else Picard)
    int schur = 0;               // pressure block of Newton solves: 0 eta_n / cell volume, 1 the Jacobian's
                                 // D11 / 2 (tangent viscosity) where positive
    // preconditioner application captured as a CUDA graph, per precision
    // ([0] FP64, [1] FP32): one graph launch per Krylov iteration
    // [precision (0 FP64, 1 FP32) * 2 + newton hierarchy + 4 * tangent Schur]
    cudaGraphExec_t pre[MDZ_PRE_SLOTS] = {};
    long long pre_launches[MDZ_PRE_SLOTS] = {};
    const double *pre_eta[MDZ_PRE_SLOTS] = {};
    double pre_bytes[MDZ_PRE_SLOTS] = {};   // algorithmic bytes of one application
};

// ---------------------------------------------------------------------------
// Tag rule of the free-slip pure-shear box on any level (the fine level must
// follow it too): Vx Dirichlet on the W/E lines, free-slip ghosts on the S/N
// rows; Vz Dirichlet on the S/N lines, ghosts on W/E; everything else inner.
__global__ void k_level_tags(int Nx, int Nz, signed char *BCu, signed char *BCv, signed char *BCp, signed char *BCg) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int nu = Nx * (Nz + 1), nv = (Nx + 1) * Nz, np = (Nx - 1) * (Nz - 1), ng = Nx * Nz;
    if (i < nu) {
        int k = i % Nx, l = i / Nx;
        signed char t = -1;
        if (k == 0 || k == Nx - 1) t = 0;
        if (l == 0 || l == Nz) t = 13;
        BCu[i] = t;
    }
    if (i < nv) {
        int k = i % (Nx + 1), l = i / (Nx + 1);
        signed char t = -1;
        if (l == 0 || l == Nz - 1) t = 0;
        if (k == 0 || k == Nx) t = 13;
        BCv[i] = t;
    }
    if (i < np) BCp[i] = -1;
    if (i < ng) BCg[i] = -1;
}

// ---------------------------------------------------------------------------
// Multigrid kernels (velocity block, Picard, homogeneous boundaries).
template <typename T>
__global__ void k_mg_diag(stokes_geom G, const T *__restrict__ D11, const T *__restrict__ D33, T *__restrict__ idu,
                          T *__restrict__ idv) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int Nx = G.Nx, Nz = G.Nz, ncx = G.ncx, nu = Nx * (Nz + 1), nv = (Nx + 1) * Nz;
    // in the level's precision, with 1/dx^2, 1/dz^2 precomputed (FP64
    // divisions are long instruction sequences on this part)
    const T celvol = gc<T>(G, GC_CELVOL), idx2 = gc<T>(G, GC_IXX), idz2 = gc<T>(G, GC_IZZ);
    if (i < nu) {
        int k = i % Nx, l = i / Nx;
        T d = 0;
        if (G.BCu[i] == -1) {
            int c2 = k - 1 + (l - 1) * ncx;
            T inS = G.BCu[i - Nx] != 13 ? T(1) : T(0), inN = G.BCu[i + Nx] != 13 ? T(1) : T(0);
            T a = (inN * D33[i] + inS * D33[i - Nx]) * idz2 + T(2.0 / 3.0) * (D11[c2 + 1] + D11[c2]) * idx2;
            d = T(1) / (a * celvol);
        }
        idu[i] = d;
    }
    if (i < nv) {
        int k = i % (Nx + 1), l = i / (Nx + 1);
        T d = 0;
        if (G.BCv[i] == -1) {
            int c1 = k + l * Nx, c2 = k - 1 + (l - 1) * ncx;
            T inW = G.BCv[i - 1] != 13 ? T(1) : T(0), inE = G.BCv[i + 1] != 13 ? T(1) : T(0);
            T a = T(2.0 / 3.0) * (D11[c2 + ncx] + D11[c2]) * idz2 + (inE * D33[c1] + inW * D33[c1 - 1]) * idx2;
            d = T(1) / (a * celvol);
        }
        idv[i] = d;
    }
}

// Prolongation weights along the "cell-centred" direction of a staggered
// component: fine line j (1..ncf) -> main coarse line and neighbour, with the
// ghost neighbour mirrored onto the main line (free slip).
__device__ __forceinline__ void cc_weights(int j, int ncc, int &J0, float &w0, int &J1, float &w1) {
    int r = j - 1, R = r >> 1;
    J0 = R + 1;
    J1 = (r & 1) ? J0 + 1 : J0 - 1;
    w0 = 0.75f; w1 = 0.25f;
    if (J1 < 1 || J1 > ncc) { w0 = 1.0f; w1 = 0.0f; J1 = J0; }
}

// Weight of coarse vertex line I for fine vertex line i (node-centred direction).
__device__ __forceinline__ float nc_weight(int i, int I) {
    if ((i & 1) == 0) return i == 2 * I ? 1.0f : 0.0f;
    return (i == 2 * I - 1 || i == 2 * I + 1) ? 0.5f : 0.0f;
}

// Unknowns under the tag rule of k_level_tags (every level of a hierarchy
// follows it; the fine level is checked before the hierarchy is built).
__device__ __forceinline__ bool u_unknown(int k, int l, int Nx, int Nz) {
    return k >= 1 && k <= Nx - 2 && l >= 1 && l <= Nz - 1;
}
__device__ __forceinline__ bool v_unknown(int i, int j, int Nx, int Nz) {
    return i >= 1 && i <= Nx - 1 && j >= 1 && j <= Nz - 2;
}

// ---------------------------------------------------------------------------
// Galerkin coarse operators.  Re-discretised coarse levels (averaged
// viscosities) lose the coupling across layers of 1e5 viscosity contrast and
// the V-cycle stops converging; R A P keeps it.  With this P (bilinear in the
// staggered sense) and R = P^T the coarse stencils close on a fixed footprint:
//   u-row (K, L):  uu  dK in [-1, 1], dL in [-2, 2]   planes  0..14: (dK+1) + 3 (dL+2)
//                  uv  I-K in [-1, 2], J-L in [-2, 1]  planes 15..30: 15 + (dI+1) + 4 (dJ+2)
//   v-row (I, J):  vv  dI in [-2, 2], dJ in [-1, 1]   planes  0..14: (dI+2) + 5 (dJ+1)
//                  vu  K-I in [-2, 1], L-J in [-1, 2]  planes 15..30: 15 + (dK+2) + 4 (dL+1)
// (u index (k, l) of the Nx x (Nz+1) box, v index (i, j) of the (Nx+1) x Nz box).
// The level-0 stencil is a subset of this footprint.

// y = A x for a stencil level, one u-row / v-row of an unknown.  The
// coefficients are loaded by a call of their own, so that a kernel can fetch
// them before it waits for the launch that writes x (the stencils change only
// in mg_setup).  Neighbours outside the box are read from the nearest line
// inside it, whose values are zero (ghost or Dirichlet nodes are never
// unknowns).  FP64 sums run in four chains: one dependent chain of 31 FP64
// multiply-adds is longer than the loads on the small levels.
template <typename T>
__device__ __forceinline__ void st_coefs(const T *s, size_t n, size_t c, T (&cf)[MG_NST]) {
#pragma unroll
    for (int q = 0; q < MG_NST; q++) cf[q] = s[(size_t)q * n + c];
}

template <typename T>
__device__ __forceinline__ T st_urow_x(int Nx, int Nz, const T (&cf)[MG_NST], const T *xu, const T *xv, int k,
                                       int l) {
    constexpr int NA = sizeof(T) == 8 ? 4 : 1;
    T s[NA] = {};
#pragma unroll
    for (int r = 0; r < 5; r++) {   // uu: (dk, dl) = (q % 3 - 1, q / 3 - 2)
        const T *p = xu + (k - 1 + min(max(l + r - 2, 0), Nz) * Nx);
#pragma unroll
        for (int d = 0; d < 3; d++) s[(3 * r + d) % NA] += cf[3 * r + d] * p[d];
    }
#pragma unroll
    for (int r = 0; r < 4; r++) {   // uv: (dI, dJ) = (q % 4 - 1, q / 4 - 2)
        const T *p = xv + (k - 1 + min(max(l + r - 2, 0), Nz - 1) * (Nx + 1));
#pragma unroll
        for (int d = 0; d < 4; d++) s[(15 + 4 * r + d) % NA] += cf[15 + 4 * r + d] * p[d];
    }
    if constexpr (NA == 4) return (s[0] + s[1]) + (s[2] + s[3]);
    else return s[0];
}

template <typename T>
__device__ __forceinline__ T st_vrow_x(int Nx, int Nz, const T (&cf)[MG_NST], const T *xu, const T *xv, int i,
                                       int j) {
    constexpr int NA = sizeof(T) == 8 ? 4 : 1;
    T s[NA] = {};
    (void)Nz;
    const int im2 = max(i - 2, 0);
#pragma unroll
    for (int r = 0; r < 3; r++) {   // vv: (dI, dJ) = (q % 5 - 2, q / 5 - 1)
        const T *p = xv + (j + r - 1) * (Nx + 1);
#pragma unroll
        for (int d = 0; d < 5; d++)
            s[(5 * r + d) % NA] += cf[5 * r + d] * p[d == 0 ? im2 : (d == 4 ? min(i + 2, Nx) : i + d - 2)];
    }
#pragma unroll
    for (int r = 0; r < 4; r++) {   // vu: (dK, dL) = (q % 4 - 2, q / 4 - 1)
        const T *p = xu + (j + r - 1) * Nx;
#pragma unroll
        for (int d = 0; d < 4; d++)
            s[(15 + 4 * r + d) % NA] += cf[15 + 4 * r + d] * p[d == 0 ? im2 : (d == 3 ? min(i + 1, Nx - 1) : i + d - 2)];
    }
    if constexpr (NA == 4) return (s[0] + s[1]) + (s[2] + s[3]);
    else return s[0];
}

template <typename T>
__device__ __forceinline__ T st_urow(int Nx, int Nz, const T *__restrict__ su, size_t nu, const T *__restrict__ xu,
                                     const T *__restrict__ xv, int k, int l) {
    T cf[MG_NST];
    st_coefs<T>(su, nu, (size_t)k + (size_t)l * Nx, cf);
    return st_urow_x<T>(Nx, Nz, cf, xu, xv, k, l);
}

template <typename T>
__device__ __forceinline__ T st_vrow(int Nx, int Nz, const T *__restrict__ sv, size_t nv, const T *__restrict__ xu,
                                     const T *__restrict__ xv, int i, int j) {
    T cf[MG_NST];
    st_coefs<T>(sv, nv, (size_t)i + (size_t)j * (Nx + 1), cf);
    return st_vrow_x<T>(Nx, Nz, cf, xu, xv, i, j);
}

template <typename T>
__global__ void k_st_diag(stokes_geom G, const T *__restrict__ su, const T *__restrict__ sv, T *__restrict__ idu,
                          T *__restrict__ idv) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    const size_t nu = (size_t)G.Nx * (G.Nz + 1), nv = (size_t)(G.Nx + 1) * G.Nz;
    if (i < (long long)nu) idu[i] = G.BCu[i] == -1 ? T(1) / su[(size_t)MG_CENTER * nu + i] : T(0);
    if (i < (long long)nv) idv[i] = G.BCv[i] == -1 ? T(1) / sv[(size_t)MG_CENTER * nv + i] : T(0);
}

#include "mg_tiles.cuh"

// Level-0 probing of the Newton block: x = indicator of the unknowns of component
// comp with (k mod 4, l mod 4) = (cx, cz); y = A x.  The operator couples a row to same-component nodes within [-1, 1]^2 and to
// other-component nodes within a 4 x 4 window, so each colour class holds at
// most one node of a row's footprint and y at the row is one coefficient.
#define MG_PROBE 4
template <typename T>
__global__ void k_probe_vec(stokes_geom G, int comp, int cx, int cz, T *__restrict__ xu, T *__restrict__ xv) {
    int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    const int Nx = G.Nx, Nz = G.Nz;
    if (i < Nx && j <= Nz) {
        int c = i + j * Nx;
        xu[c] = (comp == 0 && G.BCu[c] == -1 && i % MG_PROBE == cx && j % MG_PROBE == cz) ? T(1) : T(0);
    }
    if (i <= Nx && j < Nz) {
        int c = i + j * (Nx + 1);
        xv[c] = (comp == 1 && G.BCv[c] == -1 && i % MG_PROBE == cx && j % MG_PROBE == cz) ? T(1) : T(0);
    }
}

// velocity rows of the Newton operator applied to (xu, xv, 0); p0: a zero pressure vector
template <typename T>
__global__ void __launch_bounds__(256) k_mg_apply(stokes_geom G, stokes_coefs<T> D, const T *__restrict__ xu,
                                                  const T *__restrict__ xv, const T *__restrict__ p0,
                                                  T *__restrict__ yu, T *__restrict__ yv) {
    int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    const int Nx = G.Nx, Nz = G.Nz;
    const T celvol = gc<T>(G, GC_CELVOL);
    stokes_cvec<T> x{xu, xv, p0};
    if (i < Nx && j <= Nz) {
        int c = i + j * Nx;
        yu[c] = G.BCu[c] == -1 ? xrow<T, true>(G, D, x, i, j) * celvol : T(0);
    }
    if (i <= Nx && j < Nz) {
        int c = i + j * (Nx + 1);
        yv[c] = G.BCv[c] == -1 ? zrow<T, true>(G, D, x, i, j) * celvol : T(0);
    }
}

// offset of the colour-cx node from position p along one direction inside the
// window [lo, hi] (at most MG_PROBE wide): returns 1 and the offset, or 0
__device__ __forceinline__ int colour_offset(int p, int cx, int lo, int hi, int *d) {
    for (int o = lo; o <= hi; o++)
        if ((((p + o) % MG_PROBE) + MG_PROBE) % MG_PROBE == cx) { *d = o; return 1; }
    return 0;
}

template <typename T>
__global__ void k_probe_collect(stokes_geom G, int comp, int cx, int cz, const T *__restrict__ yu,
                                const T *__restrict__ yv, T *__restrict__ su, T *__restrict__ sv) {
    int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    const int Nx = G.Nx, Nz = G.Nz;
    const size_t nu = (size_t)Nx * (Nz + 1), nv = (size_t)(Nx + 1) * Nz;
    int a, b;
    if (i < Nx && j <= Nz) {
        int c = i + j * Nx;
        if (G.BCu[c] == -1) {
            if (comp == 0) {   // uu within [-1, 1]^2
                if (colour_offset(i, cx, -1, 1, &a) && colour_offset(j, cz, -1, 1, &b))
                    su[(size_t)((a + 1) + 3 * (b + 2)) * nu + c] = yu[c];
            } else {           // uv: I - k in [-1, 2], J - l in [-2, 1]
                if (colour_offset(i, cx, -1, 2, &a) && colour_offset(j, cz, -2, 1, &b))
                    su[(size_t)(15 + (a + 1) + 4 * (b + 2)) * nu + c] = yu[c];
            }
        }
    }
    if (i <= Nx && j < Nz) {
        int c = i + j * (Nx + 1);
        if (G.BCv[c] == -1) {
            if (comp == 1) {   // vv within [-1, 1]^2
                if (colour_offset(i, cx, -1, 1, &a) && colour_offset(j, cz, -1, 1, &b))
                    sv[(size_t)((a + 2) + 5 * (b + 1)) * nv + c] = yv[c];
            } else {           // vu: K - i in [-2, 1], L - j in [-1, 2]
                if (colour_offset(i, cx, -2, 1, &a) && colour_offset(j, cz, -1, 2, &b))
                    sv[(size_t)(15 + (a + 2) + 4 * (b + 1)) * nv + c] = yv[c];
            }
        }
    }
}

// Level-0 stencils of the Picard velocity block written out directly from
// the viscosities (the composition strain rate -> D11 / D33 stress ->
// divergence of xrow / zrow with the same row flags, times the cell volume),
// one thread per (i, j), in the level's precision; every plane of every row
// is written, zeros outside the unknowns.  Equal to probing the Picard
// operator, in one pass.
//   u-row (k, l), aE = inE D11[E], aW = inW D11[W], bN = inN D33[N], bS = inS D33[S]:
//     u(k+-1, l): -2/3 aE|aW / dx^2   u(k, l+-1): -bN|bS / dz^2   u(k, l): the sum of their negatives
//     v(k+1, l): aE/3 - bN   v(k+1, l-1): bS - aE/3   v(k, l): bN - aW/3   v(k, l-1): aW/3 - bS   (/ dx dz)
//   v-row (i, j), cN = inN D22[N], cS = inS D22[S], dE = inE D33[E], dW = inW D33[W]:
//     v(i, j+-1): -2/3 cN|cS / dz^2   v(i+-1, j): -dE|dW / dx^2   v(i, j): the sum of their negatives
//     u(i, j+1): cN/3 - dE   u(i-1, j+1): dW - cN/3   u(i, j): dE - cS/3   u(i-1, j): cS/3 - dW   (/ dx dz)
// (The free-slip box of u_unknown / v_unknown, checked before a hierarchy is
// built: every centroid and vertex is active, in* = 0 only for the shear
// stress beside a free-slip wall.)
template <typename T>
__device__ __forceinline__ void picard_coefs_u(const stokes_geom &G, const T *__restrict__ D11,
                                               const T *__restrict__ D33, int k, int l, T (&a)[MG_NST]) {
    const int Nx = G.Nx, Nz = G.Nz, c1 = k + l * Nx, c2 = k - 1 + (l - 1) * G.ncx;
    const T celvol = gc<T>(G, GC_CELVOL), ixx = gc<T>(G, GC_IXX), izz = gc<T>(G, GC_IZZ), ixz = gc<T>(G, GC_IXZ);
#pragma unroll
    for (int q = 0; q < MG_NST; q++) a[q] = T(0);
    const T aE = D11[c2 + 1], aW = D11[c2];
    const T bN = l < Nz - 1 ? D33[c1] : T(0), bS = l > 1 ? D33[c1 - Nx] : T(0);
    const T uE = -T(2.0 * T(1.0 / 3.0)) * aE * ixx, uW = -T(2.0 * T(1.0 / 3.0)) * aW * ixx;
    const T uN = -bN * izz, uS = -bS * izz;
    auto isu = [&](int kk, int ll, T v) { return u_unknown(kk, ll, Nx, Nz) ? v * celvol : T(0); };
    auto isv = [&](int ii, int jj, T v) { return v_unknown(ii, jj, Nx, Nz) ? v * celvol : T(0); };
    a[(0 + 1) + 3 * (0 + 2)] = -(uE + uW + uN + uS) * celvol;
    a[(1 + 1) + 3 * (0 + 2)] = isu(k + 1, l, uE);
    a[(-1 + 1) + 3 * (0 + 2)] = isu(k - 1, l, uW);
    a[(0 + 1) + 3 * (1 + 2)] = isu(k, l + 1, uN);
    a[(0 + 1) + 3 * (-1 + 2)] = isu(k, l - 1, uS);
    a[15 + (1 + 1) + 4 * (0 + 2)] = isv(k + 1, l, (aE * T(1.0 / 3.0) - bN) * ixz);
    a[15 + (1 + 1) + 4 * (-1 + 2)] = isv(k + 1, l - 1, (bS - aE * T(1.0 / 3.0)) * ixz);
    a[15 + (0 + 1) + 4 * (0 + 2)] = isv(k, l, (bN - aW * T(1.0 / 3.0)) * ixz);
    a[15 + (0 + 1) + 4 * (-1 + 2)] = isv(k, l - 1, (aW * T(1.0 / 3.0) - bS) * ixz);
}

template <typename T>
__device__ __forceinline__ void picard_coefs_v(const stokes_geom &G, const T *__restrict__ D11,
                                               const T *__restrict__ D33, int k, int l, T (&a)[MG_NST]) {
    const int Nx = G.Nx, Nz = G.Nz, c1 = k + l * Nx, c2 = k - 1 + (l - 1) * G.ncx;
    const T celvol = gc<T>(G, GC_CELVOL), ixx = gc<T>(G, GC_IXX), izz = gc<T>(G, GC_IZZ), ixz = gc<T>(G, GC_IXZ);
#pragma unroll
    for (int q = 0; q < MG_NST; q++) a[q] = T(0);
    const T cN = D11[c2 + G.ncx], cS = D11[c2];
    const T dE = k < Nx - 1 ? D33[c1] : T(0), dW = k > 1 ? D33[c1 - 1] : T(0);
    const T vN = -T(2.0 * T(1.0 / 3.0)) * cN * izz, vS = -T(2.0 * T(1.0 / 3.0)) * cS * izz;
    const T vE = -dE * ixx, vW = -dW * ixx;
    auto isu = [&](int kk, int ll, T v) { return u_unknown(kk, ll, Nx, Nz) ? v * celvol : T(0); };
    auto isv = [&](int ii, int jj, T v) { return v_unknown(ii, jj, Nx, Nz) ? v * celvol : T(0); };
    a[(0 + 2) + 5 * (0 + 1)] = -(vN + vS + vE + vW) * celvol;
    a[(0 + 2) + 5 * (1 + 1)] = isv(k, l + 1, vN);
    a[(0 + 2) + 5 * (-1 + 1)] = isv(k, l - 1, vS);
    a[(1 + 2) + 5 * (0 + 1)] = isv(k + 1, l, vE);
    a[(-1 + 2) + 5 * (0 + 1)] = isv(k - 1, l, vW);
    a[15 + (0 + 2) + 4 * (1 + 1)] = isu(k, l + 1, (cN * T(1.0 / 3.0) - dE) * ixz);
    a[15 + (-1 + 2) + 4 * (1 + 1)] = isu(k - 1, l + 1, (dW - cN * T(1.0 / 3.0)) * ixz);
    a[15 + (0 + 2) + 4 * (0 + 1)] = isu(k, l, (dE - cS * T(1.0 / 3.0)) * ixz);
    a[15 + (-1 + 2) + 4 * (0 + 1)] = isu(k - 1, l, (cS * T(1.0 / 3.0) - dW) * ixz);
}

template <typename T>
__global__ void __launch_bounds__(256) k_picard_stencil(stokes_geom G, const T *__restrict__ D11,
                                                        const T *__restrict__ D33, T *__restrict__ su,
                                                        T *__restrict__ sv) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    const int Nx = G.Nx, Nz = G.Nz;
    const size_t nu = (size_t)Nx * (Nz + 1), nv = (size_t)(Nx + 1) * Nz;
    T a[MG_NST];
    if (i < Nx && j <= Nz) {
        const bool unk = u_unknown(i, j, Nx, Nz);
        if (unk) picard_coefs_u<T>(G, D11, D33, i, j, a);
#pragma unroll
        for (int q = 0; q < MG_NST; q++) su[(size_t)q * nu + i + j * Nx] = unk ? a[q] : T(0);
    }
    if (i <= Nx && j < Nz) {
        const bool unk = v_unknown(i, j, Nx, Nz);
        if (unk) picard_coefs_v<T>(G, D11, D33, i, j, a);
#pragma unroll
        for (int q = 0; q < MG_NST; q++) sv[(size_t)q * nv + i + j * (Nx + 1)] = unk ? a[q] : T(0);
    }
}

// parents of fine u node (i, j) / v node (i, j) as coarse (I, J) pairs
__device__ __forceinline__ void u_parents_ij(int i, int j, int nczc, int *I, int *J, float *w) {
    int J0, J1;
    float w0, w1;
    cc_weights(j, nczc, J0, w0, J1, w1);
    const int Ia = i >> 1, Ib = (i + 1) >> 1;
    const float wa = (i & 1) ? 0.5f : 1.0f, wb = (i & 1) ? 0.5f : 0.0f;
    I[0] = Ia; J[0] = J0; w[0] = wa * w0;
    I[1] = Ia; J[1] = J1; w[1] = wa * w1;
    I[2] = Ib; J[2] = J0; w[2] = wb * w0;
    I[3] = Ib; J[3] = J1; w[3] = wb * w1;
}
__device__ __forceinline__ void v_parents_ij(int i, int j, int ncxc, int *I, int *J, float *w) {
    int I0, I1;
    float w0, w1;
    cc_weights(i, ncxc, I0, w0, I1, w1);
    const int Ja = j >> 1, Jb = (j + 1) >> 1;
    const float wa = (j & 1) ? 0.5f : 1.0f, wb = (j & 1) ? 0.5f : 0.0f;
    I[0] = I0; J[0] = Ja; w[0] = wa * w0;
    I[1] = I1; J[1] = Ja; w[1] = wa * w1;
    I[2] = I0; J[2] = Jb; w[2] = wb * w0;
    I[3] = I1; J[3] = Jb; w[3] = wb * w1;
}

// Coarse stencils = R A P.  A block forms 32 coarse rows of one component:
// each of its 12 warps takes one of the 12 fine rows a coarse row restricts
// from (3 node-centred x 4 cell-centred lines), for the 32 coarse rows of its
// lanes, so the parity of the fine indices, and with it the pattern of the
// parents, is the same across a warp; every lane accumulates its 31 entries in
// a column of shared memory of its own and the 12 columns are added up at the
// end, in warp order, together with the row's inverse diagonal.  Accumulation in
// the level's precision (FP64 throughput is a small fraction of FP32 on this
// part).  From a viscous fine level (VISC) the 9 Picard coefficients of a row are
// formed from the viscosities instead of reading 31 stored ones.  An entry
// landing outside the footprint (impossible with this P) sets *bad.
// An earlier form (four threads per coarse row, three fine rows each one
// after the other, u and v rows in the same thread) took 80-90 us on every
// level however small, and 236 us on the first level of 1025 x 513 in FP32.
#define GAL_WARPS 12
#define GAL_THREADS (32 * GAL_WARPS)
template <typename T, bool VISC>
__global__ void __launch_bounds__(GAL_THREADS) k_galerkin(stokes_geom F, const T *suF, const T *svF,
                                                          const T *__restrict__ D11,
                                                          const T *__restrict__ D33, stokes_geom Cg, int ublocks,
                                                          T *__restrict__ suC, T *__restrict__ svC,
                                                          T *__restrict__ idu, T *__restrict__ idv, int *bad) {
    extern __shared__ __align__(16) unsigned char gal_sm[];
    T *const acc_sh = reinterpret_cast<T *>(gal_sm);
    T *const acc = acc_sh + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool ublock = (int)blockIdx.x < ublocks;
    const int Nxf = F.Nx, Nzf = F.Nz, Nxc = Cg.Nx, Nzc = Cg.Nz;
    const int t0 = 32 * (ublock ? (int)blockIdx.x : (int)blockIdx.x - ublocks), t = t0 + lane;
    const int n = ublock ? Nxc * (Nzc + 1) : (Nxc + 1) * Nzc, w = ublock ? Nxc : Nxc + 1;
    const int K = t % w, L = t / w;   // coarse u node (K, L) or v node (K, L)
    const bool row = t < n && (ublock ? u_unknown(K, L, Nxc, Nzc) : v_unknown(K, L, Nxc, Nzc));
#pragma unroll
    for (int q = 0; q < MG_NST; q++) acc[q * GAL_THREADS] = T(0);
    const int cc = warp / 3, nc = warp % 3;   // cell-centred line 2 X - 2 + cc, node-centred 2 X - 1 + nc
    const float wn = nc == 1 ? 1.0f : 0.5f;
    int PI[4], PJ[4];
    float pw[4];
    T a[MG_NST];
    pdl_wait();
    auto add = [&](int slot, int di, int dj, int lo_i, int hi_i, int lo_j, int hi_j, int sd, T v) {
        if (di < lo_i || di > hi_i || dj < lo_j || dj > hi_j) { *bad = 1; return; }
        acc[(slot + (di - lo_i) + sd * (dj - lo_j)) * GAL_THREADS] += v;
    };
    if (row && ublock) {
        const int k = 2 * K - 1 + nc, l = 2 * L - 2 + cc;
        if (l >= 1 && l <= F.ncz && u_unknown(k, l, Nxf, Nzf)) {
            const T R = weight<T>(wn * cc_restrict_weight(L, cc, Cg.ncz));
            if (VISC) picard_coefs_u<T>(F, D11, D33, k, l, a);
            else st_coefs<T>(suF, (size_t)Nxf * (Nzf + 1), (size_t)k + (size_t)l * Nxf, a);
#pragma unroll
            for (int q = 0; q < 15; q++) {   // uu entries of the fine row
                if (a[q] == T(0)) continue;
                u_parents_ij(k + q % 3 - 1, l + q / 3 - 2, Cg.ncz, PI, PJ, pw);
                const T ra = R * a[q];
#pragma unroll
                for (int s = 0; s < 4; s++)
                    if (pw[s] != 0.0f && u_unknown(PI[s], PJ[s], Nxc, Nzc))
                        add(0, PI[s] - K, PJ[s] - L, -1, 1, -2, 2, 3, ra * weight<T>(pw[s]));
            }
#pragma unroll
            for (int q = 0; q < 16; q++) {   // uv entries
                if (a[15 + q] == T(0)) continue;
                v_parents_ij(k + q % 4 - 1, l + q / 4 - 2, Cg.ncx, PI, PJ, pw);
                const T ra = R * a[15 + q];
#pragma unroll
                for (int s = 0; s < 4; s++)
                    if (pw[s] != 0.0f && v_unknown(PI[s], PJ[s], Nxc, Nzc))
                        add(15, PI[s] - K, PJ[s] - L, -1, 2, -2, 1, 4, ra * weight<T>(pw[s]));
            }
        }
    } else if (row) {
        const int i = 2 * K - 2 + cc, j = 2 * L - 1 + nc;
        if (i >= 1 && i <= F.ncx && v_unknown(i, j, Nxf, Nzf)) {
            const T R = weight<T>(wn * cc_restrict_weight(K, cc, Cg.ncx));
            if (VISC) picard_coefs_v<T>(F, D11, D33, i, j, a);
            else st_coefs<T>(svF, (size_t)(Nxf + 1) * Nzf, (size_t)i + (size_t)j * (Nxf + 1), a);
#pragma unroll
            for (int q = 0; q < 15; q++) {   // vv entries
                if (a[q] == T(0)) continue;
                v_parents_ij(i + q % 5 - 2, j + q / 5 - 1, Cg.ncx, PI, PJ, pw);
                const T ra = R * a[q];
#pragma unroll
                for (int s = 0; s < 4; s++)
                    if (pw[s] != 0.0f && v_unknown(PI[s], PJ[s], Nxc, Nzc))
                        add(0, PI[s] - K, PJ[s] - L, -2, 2, -1, 1, 5, ra * weight<T>(pw[s]));
            }
#pragma unroll
            for (int q = 0; q < 16; q++) {   // vu entries
                if (a[15 + q] == T(0)) continue;
                u_parents_ij(i + q % 4 - 2, j + q / 4 - 1, Cg.ncz, PI, PJ, pw);
                const T ra = R * a[15 + q];
#pragma unroll
                for (int s = 0; s < 4; s++)
                    if (pw[s] != 0.0f && u_unknown(PI[s], PJ[s], Nxc, Nzc))
                        add(15, PI[s] - K, PJ[s] - L, -2, 1, -1, 2, 4, ra * weight<T>(pw[s]));
            }
        }
    }
    __syncthreads();
    T *out = ublock ? suC : svC, *id = ublock ? idu : idv;
    for (int q = warp; q < MG_NST; q += GAL_WARPS) {
        if (t >= n) continue;
        const T *c = acc_sh + q * GAL_THREADS + lane;
        T s = 0;
#pragma unroll
        for (int e = 0; e < GAL_WARPS; e++) s += c[32 * e];
        out[(size_t)q * n + t] = s;
        if (q == MG_CENTER) id[t] = row ? T(1) / s : T(0);
    }
}

template <typename T>
__global__ void k_fill_D11_D33(int nc, int nv, const double *__restrict__ eta_n, const double *__restrict__ eta_s,
                               T *__restrict__ D11, T *__restrict__ D33) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nc) D11[i] = (T)(2.0 * eta_n[i]);
    if (i < nv) D33[i] = (T)eta_s[i];
}

// ---------------------------------------------------------------------------
// Coarsest level: one CTA runs Jacobi-preconditioned CG on the whole level.
template <typename T>
__device__ double cta_dot(const T *a, const T *b, int n0, int n1, const T *a1, const T *b1, double *sh) {
    double s = 0.0;
    for (int i = threadIdx.x; i < n0; i += blockDim.x) s += (double)a[i] * (double)b[i];
    for (int i = threadIdx.x; i < n1; i += blockDim.x) s += (double)a1[i] * (double)b1[i];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) sh[wid] = s;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x < 32) {
        t = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (threadIdx.x == 0) sh[32] = t;
    }
    __syncthreads();
    return sh[32];
}

template <typename T>
__device__ void cta_apply(const stokes_geom &G, const T *su, const T *sv, const T *xu, const T *xv, T *yu, T *yv) {
    const int Nx = G.Nx, Nz = G.Nz;
    const size_t nu = (size_t)Nx * (Nz + 1), nv = (size_t)(Nx + 1) * Nz;
    for (int c = threadIdx.x; c < (int)nu; c += blockDim.x)
        yu[c] = G.BCu[c] == -1 ? st_urow<T>(Nx, Nz, su, nu, xu, xv, c % Nx, c / Nx) : T(0);
    for (int c = threadIdx.x; c < (int)nv; c += blockDim.x)
        yv[c] = G.BCv[c] == -1 ? st_vrow<T>(Nx, Nz, sv, nv, xu, xv, c % (Nx + 1), c / (Nx + 1)) : T(0);
}

template <typename T>
__global__ void __launch_bounds__(1024) k_mg_coarse_cg(stokes_geom G, const T *su, const T *sv, const T *__restrict__ fu,
                                                       const T *__restrict__ fv, const T *__restrict__ idu,
                                                       const T *__restrict__ idv, T *xu, T *xv, T *ru, T *rv, T *zu,
                                                       T *zv, T *pu, T *pv, T *qu, T *qv, int maxit, double rtol) {
    __shared__ double sh[34];
    const int nu = G.Nx * (G.Nz + 1), nv = (G.Nx + 1) * G.Nz;
    for (int i = threadIdx.x; i < nu; i += blockDim.x) { xu[i] = 0; ru[i] = fu[i]; zu[i] = idu[i] * fu[i]; pu[i] = zu[i]; }
    for (int i = threadIdx.x; i < nv; i += blockDim.x) { xv[i] = 0; rv[i] = fv[i]; zv[i] = idv[i] * fv[i]; pv[i] = zv[i]; }
    __syncthreads();
    double rz = cta_dot<T>(ru, zu, nu, nv, rv, zv, sh);
    double r0 = cta_dot<T>(ru, ru, nu, nv, rv, rv, sh);
    if (r0 == 0.0) return;
    for (int it = 0; it < maxit; it++) {
        cta_apply<T>(G, su, sv, pu, pv, qu, qv);
        __syncthreads();
        double pq = cta_dot<T>(pu, qu, nu, nv, pv, qv, sh);
        if (pq <= 0.0) break;
        T a = (T)(rz / pq);
        for (int i = threadIdx.x; i < nu; i += blockDim.x) { xu[i] += a * pu[i]; ru[i] -= a * qu[i]; zu[i] = idu[i] * ru[i]; }
        for (int i = threadIdx.x; i < nv; i += blockDim.x) { xv[i] += a * pv[i]; rv[i] -= a * qv[i]; zv[i] = idv[i] * rv[i]; }
        __syncthreads();
        double rz1 = cta_dot<T>(ru, zu, nu, nv, rv, zv, sh);
        double rr = cta_dot<T>(ru, ru, nu, nv, rv, rv, sh);
        if (rr <= rtol * rtol * r0) break;
        T b = (T)(rz1 / rz);
        rz = rz1;
        for (int i = threadIdx.x; i < nu; i += blockDim.x) pu[i] = zu[i] + b * pu[i];
        for (int i = threadIdx.x; i < nv; i += blockDim.x) pv[i] = zv[i] + b * pv[i];
        __syncthreads();
    }
}

// Small coarsest level: the velocity block is gathered from the level's
// stencils into a dense matrix (one CTA) and inverted by Gauss-Jordan
// elimination with partial pivoting (a zero pivot column sets *status).  AinvT is stored column-major so that the solve's threads read it
// coalesced.  Dense numbering: u unknowns (k, l), k in 1..Nx-2, l in 1..Nz-1,
// row by row, then v unknowns (i, j), i in 1..Nx-1, j in 1..Nz-2.
__device__ __forceinline__ int dense_u(int Nx, int Nz, int k, int l) {
    return (k >= 1 && k <= Nx - 2 && l >= 1 && l <= Nz - 1) ? (k - 1) + (l - 1) * (Nx - 2) : -1;
}
__device__ __forceinline__ int dense_v(int Nx, int Nz, int i, int j) {
    return (i >= 1 && i <= Nx - 1 && j >= 1 && j <= Nz - 2) ? (Nx - 2) * (Nz - 1) + (i - 1) + (j - 1) * (Nx - 1) : -1;
}

// In the hierarchy's precision: the FP32 hierarchy's inverse is stored in FP32
// and only corrects a V-cycle.  In place (the pivot column's slot takes the
// inverse's), in shared memory where it fits (the launch passes the dynamic
// size), else in the global work array; per step one warp finds the pivot and
// its reciprocal, then the pivot row and column are copied, then every element
// is updated: three barriers.  (Eliminating [A | I] with seven barriers and a
// division per thread and step took 300 us in FP64 and 155 us in FP32 for the
// 52 unknowns of 8 x 4 cells.)
template <typename T>
__global__ void __launch_bounds__(512) k_coarse_dense_setup(stokes_geom G, const T *__restrict__ su,
                                                            const T *__restrict__ sv, int n,
                                                            const int *__restrict__ map, T *Ag,
                                                            T *__restrict__ AinvT, int *status) {
    extern __shared__ __align__(16) unsigned char dsm[];
    T *A = (size_t)n * n * sizeof(T) <= MG_DENSE_SMEM ? reinterpret_cast<T *>(dsm) : Ag;
    __shared__ T prow[MG_DENSE_MAX], col[MG_DENSE_MAX], s_inv;
    __shared__ int perm[MG_DENSE_MAX], s_pr;
    const int Nx = G.Nx, Nz = G.Nz, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
    const size_t nu = (size_t)Nx * (Nz + 1), nv = (size_t)(Nx + 1) * Nz;
    for (int e = tid; e < n * n; e += blockDim.x) A[e] = T(0);
    __syncthreads();
    for (int r = tid; r < n; r += blockDim.x) {
        const int m = map[r];
        if (m < (int)nu) {
            const int k = m % Nx, l = m / Nx;
            for (int q = 0; q < 15; q++) {
                int c = dense_u(Nx, Nz, k + q % 3 - 1, l + q / 3 - 2);
                if (c >= 0) A[(size_t)r * n + c] += su[(size_t)q * nu + m];
            }
            for (int q = 0; q < 16; q++) {
                int c = dense_v(Nx, Nz, k + q % 4 - 1, l + q / 4 - 2);
                if (c >= 0) A[(size_t)r * n + c] += su[(size_t)(15 + q) * nu + m];
            }
        } else {
            const int mv = m - (int)nu, i = mv % (Nx + 1), j = mv / (Nx + 1);
            for (int q = 0; q < 15; q++) {
                int c = dense_v(Nx, Nz, i + q % 5 - 2, j + q / 5 - 1);
                if (c >= 0) A[(size_t)r * n + c] += sv[(size_t)q * nv + mv];
            }
            for (int q = 0; q < 16; q++) {
                int c = dense_u(Nx, Nz, i + q % 4 - 2, j + q / 4 - 1);
                if (c >= 0) A[(size_t)r * n + c] += sv[(size_t)(15 + q) * nv + mv];
            }
        }
    }
    __syncthreads();
    // Gauss-Jordan with partial pivoting (the Newton block is neither
    // symmetric nor definite)
    for (int k = 0; k < n; k++) {
        if (wid == 0) {
            T bv = T(-1);
            int bi = k;
            for (int i = k + lane; i < n; i += 32) {
                const T v = fabs(A[(size_t)i * n + k]);
                if (v > bv) { bv = v; bi = i; }
            }
            for (int o = 16; o > 0; o >>= 1) {
                const T ov = __shfl_xor_sync(0xffffffffu, bv, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
            }
            if (lane == 0) {
                const bool ok = bv > T(0) && isfinite(bv);
                s_pr = ok ? bi : -1;
                s_inv = ok ? T(1) / A[(size_t)bi * n + k] : T(0);
            }
        }
        __syncthreads();
        const int pr = s_pr;
        const T inv = s_inv;
        if (pr < 0) {   // uniform
            if (tid == 0) *status = 1;
            return;
        }
        for (int j = tid; j < n; j += blockDim.x) {
            const T ap = A[(size_t)pr * n + j], ak = A[(size_t)k * n + j];
            prow[j] = j == k ? inv : ap * inv;
            col[j] = j == pr ? A[(size_t)k * n + k] : A[(size_t)j * n + k];
            if (j == 0) perm[k] = pr;
            if (pr != k && j != k) A[(size_t)pr * n + j] = ak;   // (column k is rewritten below)
        }
        __syncthreads();
        for (int i = wid; i < n; i += nw) {
            const T c = col[i];
            for (int j = lane; j < n; j += 32) {
                T *a = A + (size_t)i * n + j;
                *a = i == k ? prow[j] : (j == k ? T(0) : *a) - c * prow[j];
            }
        }
        __syncthreads();
    }
    // the row interchanges become column interchanges of the inverse, last first
    int *src = reinterpret_cast<int *>(col);
    for (int j = tid; j < n; j += blockDim.x) src[j] = j;
    __syncthreads();
    if (tid == 0)
        for (int k = n - 1; k >= 0; k--) { const int t = src[k]; src[k] = src[perm[k]]; src[perm[k]] = t; }
    __syncthreads();
    for (int e = tid; e < n * n; e += blockDim.x) {
        const int i = e / n, j = e % n;
        AinvT[(size_t)j * n + i] = A[(size_t)i * n + src[j]];
    }
}

// x = A^-1 f on the small coarsest level (zero outside the unknowns): eight
// lanes per row, so that the row's products are not one chain of loads
template <typename T>
__device__ __forceinline__ T dense_row(int n, const T *AinvT, const T *fs, int r, int lane) {
    T s = 0;
    if (r < n)
        for (int j = lane; j < n; j += 8) s += AinvT[(size_t)j * n + r] * fs[j];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

template <typename T>
__global__ void __launch_bounds__(512) k_coarse_dense_solve(int n, int nu, int nv, const int *__restrict__ map,
                                                            const T *__restrict__ AinvT, const T *fu, const T *fv,
                                                            T *__restrict__ xu, T *__restrict__ xv) {
    __shared__ T fs[MG_DENSE_MAX];
    mg_release<T>();
    pdl_wait();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        int m = map[i];
        fs[i] = m < nu ? fu[m] : fv[m - nu];
    }
    for (int i = threadIdx.x; i < nu; i += blockDim.x) xu[i] = T(0);
    for (int i = threadIdx.x; i < nv; i += blockDim.x) xv[i] = T(0);
    __syncthreads();
    for (int r0 = 0; r0 < n; r0 += blockDim.x / 8) {
        const int r = r0 + threadIdx.x / 8;
        const T s = dense_row<T>(n, AinvT, fs, r, threadIdx.x & 7);
        if (r < n && (threadIdx.x & 7) == 0) {
            const int m = map[r];
            if (m < nu) xu[m] = s; else xv[m - nu] = s;
        }
    }
}

// ---------------------------------------------------------------------------
// Bottom of the V-cycle in one cluster of 8 CTAs, everything in shared memory.
// As grid kernels the smallest levels cost one launch per phase, several
// microseconds for a few hundred rows.  Here each CTA copies the stencils and
// inverse diagonals of its eighth of every level's unknown rows, and its rows of
// the coarsest inverse, into shared memory before it waits for the launch that
// writes the right-hand side.  The vectors are held whole in every CTA: a phase
// computes the own rows from them and stores the results into all eight
// (st.shared::cluster), then the cluster meets.  Right-hand sides are needed on
// the own rows only, and restriction writes the next level's first sweep.
//
// In FP64 a warp instruction takes its scheduler's unit 64 clocks, so a phase of
// one warp is 36 x 64: where a CTA has few rows (MG_BOTTOM_SPLIT) four lanes
// share one, in the four chains of the row functions (the same bits).  The
// kernel before releases it at once, so that the stencils are loaded meanwhile
// (6000 clocks); a phase is then 1000 to 3700 clocks and a meeting 1000.
//
// One CTA for all rows could take levels of up to 256 rows in FP64 (16.5 to
// 21 us), every level above being three launches.  V-cycle, 8 CTAs after one:
// 100 x 100 cells 85 -> 73 us, 120 x 60 73 -> 65, 256 x 128 94 -> 80, 400 x 400
// 197 -> 184, 1024 x 512 in FP32 111 -> 109; with 16 CTAs 78, 67, 84, 190, 116,
// with 4 79, 69, 87, 190, 109.  A cluster of 16 CTAs out of L2 (no shared
// memory) took 89 us for 128 x 64 cells in FP32 and 203 us in FP64.
#define MG_BOTTOM_MAX 6
#define MG_BOTTOM_CTAS 8
#define MG_BOTTOM_SMEM (200 * 1024)
#define MG_BOTTOM_SPLIT 96   // FP64 rows per CTA up to which four lanes share a row
template <typename T>
constexpr int mg_bottom_threads() { return sizeof(T) == 8 ? 256 : 512; }
template <typename T>
struct mg_bottom_args {
    int nlev, nu1, nu2, ndense;   // nlev levels, the last one the dense coarsest
    T omega;
    const int *dmap;
    const T *AinvT;
    int Nx[MG_BOTTOM_MAX], Nz[MG_BOTTOM_MAX];
    const T *su[MG_BOTTOM_MAX], *sv[MG_BOTTOM_MAX], *idu[MG_BOTTOM_MAX], *idv[MG_BOTTOM_MAX];
    const T *fu, *fv;             // right-hand side of the first level
    T *xu, *xv;                   // its result
};

__host__ __device__ inline int mg_bottom_rows_u(int Nx, int Nz) { return (Nx - 2) * (Nz - 1); }
__host__ __device__ inline int mg_bottom_rows_v(int Nx, int Nz) { return (Nx - 1) * (Nz - 2); }
__host__ __device__ inline int mg_bottom_rows(int Nx, int Nz) { return mg_bottom_rows_u(Nx, Nz) + mg_bottom_rows_v(Nx, Nz); }
__host__ __device__ inline int mg_bottom_box(int Nx, int Nz) { return Nx * (Nz + 1) + (Nx + 1) * Nz; }
__host__ __device__ inline int mg_bottom_share(int rows) { return (rows + MG_BOTTOM_CTAS - 1) / MG_BOTTOM_CTAS; }
// elements of one level in a CTA: vectors x and y (also the residual) in box
// layout, then coefficients, inverse diagonal and f of its rows
__host__ __device__ inline int mg_bottom_level_elems(int Nx, int Nz) {
    return 2 * mg_bottom_box(Nx, Nz) +
           (MG_NST + 2) * (mg_bottom_share(mg_bottom_rows_u(Nx, Nz)) + mg_bottom_share(mg_bottom_rows_v(Nx, Nz)));
}
// A CTA's rows of a level: `Su` u rows, then v rows, S places in all.  Rows
// meet threads by index: u rows, a gap up to a multiple of `align`, v rows, so
// that no warp holds both kinds.
struct mg_bottom_rank {
    int Nx, Nz, Ru, Rv, Su, S, box, nu, rank;
    __device__ __forceinline__ mg_bottom_rank(int Nx_, int Nz_, int rank_) : Nx(Nx_), Nz(Nz_), rank(rank_) {
        Ru = mg_bottom_rows_u(Nx, Nz);
        Rv = mg_bottom_rows_v(Nx, Nz);
        Su = mg_bottom_share(Ru);
        S = Su + mg_bottom_share(Rv);
        box = mg_bottom_box(Nx, Nz);
        nu = Nx * (Nz + 1);
    }
    __device__ __forceinline__ int count(int align) const { return (Su + align - 1) / align * align + S - Su; }
    // row of index t: its place i among the CTA's rows, (k, j) and place in the box; false: none
    __device__ __forceinline__ bool row(int t, int align, bool &u, int &i, int &k, int &j, int &c) const {
        const int gap = (Su + align - 1) / align * align;
        u = t < gap;
        i = u ? t : Su + t - gap;
        const int r = u ? rank * Su + t : rank * (S - Su) + t - gap, w = u ? Nx - 2 : Nx - 1;
        k = 1 + r % w;
        j = 1 + r / w;
        c = u ? k + j * Nx : nu + k + j * (Nx + 1);
        return u ? t < Su && r < Ru : t - gap < S - Su && r < Rv;
    }
};

// Quarter s of row (k, j)'s product: coefficients s, s + 4, ... (the chains of
// st_urow_x and st_vrow_x in FP64)
template <typename T>
__device__ __forceinline__ T st_row_quarter(bool u, int Nx, int Nz, const T *cf, int S, const T *x, int k, int j, int s) {
    const T *const xv = x + Nx * (Nz + 1);
    T a = 0;
#pragma unroll
    for (int t = 0; t < 8; t++) {
        const int q = 4 * t + s;
        if (q >= MG_NST) break;
        const T *p;
        if (q < 15) {
            const int w = u ? 3 : 5, r = q / w, d = q - w * r;
            if (u) p = x + (k - 1 + d) + min(max(j + r - 2, 0), Nz) * Nx;
            else p = xv + (j + r - 1) * (Nx + 1) + min(max(k + d - 2, 0), Nx);
        } else {
            const int r = (q - 15) >> 2, d = (q - 15) & 3;
            if (u) p = xv + (k - 1 + d) + min(max(j + r - 2, 0), Nz - 1) * (Nx + 1);
            else p = x + (j + r - 1) * Nx + min(max(k + d - 2, 0), Nx - 1);
        }
        a += cf[q * S] * *p;
    }
    return a;
}

__device__ __forceinline__ void cluster_meet() {
    __syncwarp();   // (.aligned: the lanes of a warp arrive together)
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void st_cluster(uint32_t a, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void st_cluster(uint32_t a, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}

template <typename T>
__global__ void __launch_bounds__(mg_bottom_threads<T>()) k_mg_bottom(const __grid_constant__ mg_bottom_args<T> A) {
    extern __shared__ __align__(16) unsigned char bottom_sm[];
    T *const sm = reinterpret_cast<T *>(bottom_sm);
    mg_release<T>();
    constexpr int NT = mg_bottom_threads<T>(), C = MG_BOTTOM_CTAS;
    const int tid = threadIdx.x, lc = A.nlev - 1, n = A.ndense;
    const int rank = blockIdx.x;   // the grid is the one cluster
    uint32_t remote[C];            // the CTAs' shared memory in the cluster's address window
#pragma unroll
    for (int c = 0; c < C; c++)
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                     : "=r"(remote[c])
                     : "r"((uint32_t)__cvta_generic_to_shared(sm)), "r"(c));
    auto put = [&](T *p, T v) {    // into this place of every CTA
        const uint32_t o = (uint32_t)((p - sm) * sizeof(T));
#pragma unroll
        for (int c = 0; c < C; c++) st_cluster(remote[c] + o, v);
    };
    // ---- static data, while the launch before is still running
    int off = 0;
    for (int l = 0; l < lc; l++) {
        const mg_bottom_rank L(A.Nx[l], A.Nz[l], rank);
        const size_t nu = L.nu, nv = (size_t)(L.Nx + 1) * L.Nz;
        T *vec = sm + off, *cf0 = vec + 2 * L.box;
        for (int t = tid; t < L.count(32); t += NT) {
            bool u;
            int i, k, j, b;
            if (!L.row(t, 32, u, i, k, j, b)) continue;
            const size_t c = u ? (size_t)b : (size_t)b - nu;
            T cf[MG_NST];
            st_coefs<T>(u ? A.su[l] : A.sv[l], u ? nu : nv, c, cf);
#pragma unroll
            for (int e = 0; e < MG_NST; e++) cf0[e * L.S + i] = cf[e];
            cf0[MG_NST * L.S + i] = u ? A.idu[l][c] : A.idv[l][c];
        }
        for (int e = tid; e < 2 * L.box; e += NT) vec[e] = T(0);
        off += mg_bottom_level_elems(L.Nx, L.Nz);
    }
    const int cbox = mg_bottom_box(A.Nx[lc], A.Nz[lc]), Sn = mg_bottom_share(n), n0 = rank * Sn,
              nown = n - n0 < Sn ? n - n0 : Sn;   // dense rows of this CTA (none: <= 0)
    T *const cx = sm + off, *const fs = cx + cbox, *const Ai = fs + n;
    for (int e = tid; e < cbox; e += NT) cx[e] = T(0);
    for (int e = tid; e < n * Sn; e += NT) {
        const int i = e % Sn;
        if (i < nown) Ai[e] = A.AinvT[(size_t)(e / Sn) * n + n0 + i];
    }
    cluster_meet();   // every CTA has cleared its vectors before any stores into them
    pdl_wait();
    {   // the caller's vectors are 0 where there is no unknown
        const mg_bottom_rank L(A.Nx[0], A.Nz[0], rank);
        for (int e = rank * NT + tid; e < L.box; e += C * NT) {
            const bool u = e < L.nu;
            const int k = u ? e % L.Nx : (e - L.nu) % (L.Nx + 1), j = u ? e / L.Nx : (e - L.nu) / (L.Nx + 1);
            if (u && !(k > 0 && k < L.Nx - 1 && j > 0 && j < L.Nz)) A.xu[e] = T(0);
            if (!u && !(k > 0 && k < L.Nx && j > 0 && j < L.Nz - 1)) A.xv[e - L.nu] = T(0);
        }
    }
    unsigned par = 0;   // bit l: level l's x is in its second vector
    // mode 1: y = x + omega D^-1 (f - A x); 2: y = f - A x; 3: as 1, into the caller's vectors
    auto rows = [&](int base, int l, bool odd, int mode) {
        const mg_bottom_rank L(A.Nx[l], A.Nz[l], rank);
        T *const x = sm + base + (odd ? L.box : 0), *const y = sm + base + (odd ? 0 : L.box),
                 *const cf0 = sm + base + 2 * L.box;
        bool u;
        int i, k, j, c;
        if (sizeof(T) == 8 && L.count(8) <= MG_BOTTOM_SPLIT) {   // four lanes per row
            const int s = tid & 3;
            for (int t = tid >> 2; t < (L.count(8) + 7) / 8 * 8; t += NT / 4) {
                const bool in = L.row(t, 8, u, i, k, j, c);
                T ax = in ? st_row_quarter<T>(u, L.Nx, L.Nz, cf0 + i, L.S, x, k, j, s) : T(0);
                ax += __shfl_xor_sync(0xffffffffu, ax, 1);
                ax += __shfl_xor_sync(0xffffffffu, ax, 2);
                if (!in) continue;
                const T r = cf0[(MG_NST + 1) * L.S + i] - ax;
                const T v = mode == 2 ? r : x[c] + A.omega * cf0[MG_NST * L.S + i] * r;
                if (mode != 3) {   // into two CTAs each
                    const uint32_t o = (uint32_t)((y + c - sm) * sizeof(T));
#pragma unroll
                    for (int q = 0; q < C; q++)
                        if ((q & 3) == s) st_cluster(remote[q] + o, v);
                } else if (s == 0) {
                    if (u) A.xu[c] = v;
                    else A.xv[c - L.nu] = v;
                }
            }
        } else {
            for (int t = tid; t < L.count(32); t += NT) {
                if (!L.row(t, 32, u, i, k, j, c)) continue;
                T cf[MG_NST];
#pragma unroll
                for (int e = 0; e < MG_NST; e++) cf[e] = cf0[e * L.S + i];
                const T ax = u ? st_urow_x<T>(L.Nx, L.Nz, cf, x, x + L.nu, k, j)
                               : st_vrow_x<T>(L.Nx, L.Nz, cf, x, x + L.nu, k, j);
                const T r = cf0[(MG_NST + 1) * L.S + i] - ax;
                const T v = mode == 2 ? r : x[c] + A.omega * cf0[MG_NST * L.S + i] * r;
                if (mode != 3) put(y + c, v);
                else if (u) A.xu[c] = v;
                else A.xv[c - L.nu] = v;
            }
        }
        if (mode != 3) cluster_meet();
    };
    int base = 0;
    {   // right-hand side of the own rows and the first sweep from x = 0
        const mg_bottom_rank L(A.Nx[0], A.Nz[0], rank);
        T *const cf0 = sm + 2 * L.box;
        for (int t = tid; t < L.count(32); t += NT) {
            bool u;
            int i, k, j, c;
            if (!L.row(t, 32, u, i, k, j, c)) continue;
            const T f = u ? A.fu[c] : A.fv[c - L.nu];
            cf0[(MG_NST + 1) * L.S + i] = f;
            put(sm + c, A.omega * cf0[MG_NST * L.S + i] * f);
        }
        cluster_meet();
    }
    for (int l = 0; l < lc; l++) {
        const int Nx = A.Nx[l], Nz = A.Nz[l], next = base + mg_bottom_level_elems(Nx, Nz);
        bool odd = false;
        for (int s = 1; s < A.nu1; s++) { rows(base, l, odd, 1); odd = !odd; }
        if (odd) par |= 1u << l;
        rows(base, l, odd, 2);
        // restriction of the residual
        const box_geom F{Nx, Nz, Nx - 1, Nz - 1}, Cg{A.Nx[l + 1], A.Nz[l + 1], A.Nx[l + 1] - 1, A.Nz[l + 1] - 1};
        const T *r = sm + base + (odd ? 0 : mg_bottom_box(Nx, Nz)), *rv = r + Nx * (Nz + 1);
        if (l + 1 < lc) {   // and the next level's first sweep
            const mg_bottom_rank L(Cg.Nx, Cg.Nz, rank);
            T *const cf0 = sm + next + 2 * L.box;
            for (int t = tid; t < L.count(32); t += NT) {
                bool u;
                int i, I, J, c;
                if (!L.row(t, 32, u, i, I, J, c)) continue;
                const T f = u ? restricted_u<T>(F, Cg, r, I, J) : restricted_v<T>(F, Cg, rv, I, J);
                cf0[(MG_NST + 1) * L.S + i] = f;
                put(sm + next + c, A.omega * cf0[MG_NST * L.S + i] * f);
            }
        } else {
            const int nuc = Cg.Nx * (Cg.Nz + 1);
            for (int i = tid; i < nown; i += NT) {
                const int m = A.dmap[n0 + i], q = m - nuc;
                put(fs + n0 + i, m < nuc ? restricted_u<T>(F, Cg, r, m % Cg.Nx, m / Cg.Nx)
                                         : restricted_v<T>(F, Cg, rv, q % (Cg.Nx + 1), q / (Cg.Nx + 1)));
            }
        }
        cluster_meet();
        base = next;
    }
    // coarsest level: x = A^-1 f, eight lanes per row
    for (int r0 = 0; r0 < nown; r0 += NT / 8) {
        const int r = r0 + tid / 8;
        T s = 0;
        if (r < nown)
            for (int j = tid & 7; j < n; j += 8) s += Ai[j * Sn + r] * fs[j];
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (r < nown && (tid & 7) == 0) put(cx + A.dmap[n0 + r], s);
    }
    cluster_meet();
    for (int l = lc - 1; l >= 0; l--) {
        const int Nx = A.Nx[l], Nz = A.Nz[l], next = base;
        base -= mg_bottom_level_elems(Nx, Nz);
        bool odd = par >> l & 1;
        const box_geom F{Nx, Nz, Nx - 1, Nz - 1}, Cg{A.Nx[l + 1], A.Nz[l + 1], A.Nx[l + 1] - 1, A.Nz[l + 1] - 1};
        const mg_bottom_rank L(Nx, Nz, rank);
        const int nuc = Cg.Nx * (Cg.Nz + 1);
        T *x = sm + base + (odd ? L.box : 0);
        const T *c = sm + next + (par >> (l + 1) & 1 ? mg_bottom_box(Cg.Nx, Cg.Nz) : 0);
        const bool last = l == 0 && A.nu2 == 0;
        for (int t = tid; t < L.count(32); t += NT) {
            bool u;
            int i, k, j, b;
            if (!L.row(t, 32, u, i, k, j, b)) continue;
            const T v = u ? prolonged_u<T>(F, Cg, c, x, k, j) : prolonged_v<T>(F, Cg, c + nuc, x + L.nu, k, j);
            if (!last) put(x + b, v);
            else if (u) A.xu[b] = v;
            else A.xv[b - L.nu] = v;
        }
        if (last) break;
        cluster_meet();
        for (int s = 0; s < A.nu2; s++) {
            rows(base, l, odd, l == 0 && s == A.nu2 - 1 ? 3 : 1);
            odd = !odd;
        }
        par = odd ? par | 1u << l : par & ~(1u << l);
    }
}

// Whether the device, or the part of it that the process has, can place the
// bottom's cluster at its largest; else every level runs as launches of its own.
template <typename T>
static bool mg_bottom_placed() {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(MG_BOTTOM_CTAS);
    cfg.blockDim = dim3(mg_bottom_threads<T>());
    cfg.dynamicSmemBytes = MG_BOTTOM_SMEM;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = MG_BOTTOM_CTAS;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(k_mg_bottom<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, MG_BOTTOM_SMEM) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&n, k_mg_bottom<T>, &cfg) == cudaSuccess)
        return n >= 1;
    (void)cudaGetLastError();
    return false;
}

// ---------------------------------------------------------------------------
template <typename T>
static cudaError_t alloc0(T **p, size_t n) {
    cudaError_t e = cudaMalloc((void **)p, sizeof(T) * (n ? n : 1));
    if (e == cudaSuccess) e = cudaMemset(*p, 0, sizeof(T) * (n ? n : 1));
    return e;
}

template <typename T>
static mdz_status build_hierarchy(mdz_ctx *ctx, mg_hier<T> &H) {
    const mdz_dgrid &g = ctx->g;
    int Nx = g.Nx, Nz = g.Nz;
    double dx = g.dx, dz = g.dz;
    cudaError_t e = cudaSuccess;
    int lev = 0;
    while (lev < MG_MAX_LEVELS) {
        mg_level<T> &L = H.L[lev];
        L.Nx = Nx; L.Nz = Nz; L.ncx = Nx - 1; L.ncz = Nz - 1; L.dx = dx; L.dz = dz;
        if (lev == 0) {
            L.BCu = g.BCu; L.BCv = g.BCv; L.BCp = g.BCp; L.BCg = g.BCg; L.own_tags = false;
        } else {
            L.own_tags = true;
            if (e == cudaSuccess) e = alloc0(&L.BCu, L.nu());
            if (e == cudaSuccess) e = alloc0(&L.BCv, L.nv());
            if (e == cudaSuccess) e = alloc0(&L.BCp, (size_t)L.ncx * L.ncz);
            if (e == cudaSuccess) e = alloc0(&L.BCg, (size_t)Nx * Nz);
            if (e == cudaSuccess) {
                k_level_tags<<<mdz_blocks((size_t)(Nx + 1) * (Nz + 1)), MDZ_THREADS>>>(Nx, Nz, L.BCu, L.BCv, L.BCp, L.BCg);
                e = cudaGetLastError();
            }
        }
        if (lev == 0) {
            if (e == cudaSuccess) e = alloc0(&L.D11, (size_t)L.ncx * L.ncz);
            if (e == cudaSuccess) e = alloc0(&L.D33, (size_t)Nx * Nz);
            if (e == cudaSuccess) e = alloc0(&L.pz, (size_t)L.ncx * L.ncz);
            if (e == cudaSuccess) e = alloc0(&H.pmean, 4);
        }
        if (e == cudaSuccess) e = alloc0(&L.su, (size_t)MG_NST * L.nu());
        if (e == cudaSuccess) e = alloc0(&L.sv, (size_t)MG_NST * L.nv());
        T **bufs[] = {&L.xu, &L.yu, &L.fu, &L.ru, &L.idu};
        for (T **b : bufs) if (e == cudaSuccess) e = alloc0(b, L.nu());
        T **bufv[] = {&L.xv, &L.yv, &L.fv, &L.rv, &L.idv};
        for (T **b : bufv) if (e == cudaSuccess) e = alloc0(b, L.nv());
        lev++;
        // halve while the coarse level keeps >= 4 cells a side.  An odd cell
        // count is halved rounding up: the last coarse cell then covers one fine
        // cell, its far wall lies one fine cell outside the box, and the fine
        // points that would lie beyond the wall are not unknowns, so P and the
        // Galerkin product keep their index arithmetic and footprint.
        // (k_mg_coarse_cg, the one-CTA conjugate gradients of a coarsest level
        // too large for the dense inverse, took 2.2 ms of every FP64 V-cycle on
        // the 25 x 25 cells a 401^2 box used to end in, against 0.2 ms for the
        // levels that replace it: 101^2 defect solve 225 -> 16.2 ms, 401^2
        // shear-band step 310 -> 104 ms.  It is left for boxes some four times
        // longer than high and more.)
        const int cx = (L.ncx + 1) / 2, cz = (L.ncz + 1) / 2;
        if (cx < 4 || cz < 4) break;
        Nx = cx + 1; Nz = cz + 1; dx *= 2; dz *= 2;
    }
    H.nlev = lev;
    mg_level<T> &C = H.L[lev - 1];
    // unknowns of the coarsest level (tag rule of the free-slip box)
    std::vector<int> map;
    for (int l = 1; l <= C.Nz - 1; l++)
        for (int k = 1; k <= C.Nx - 2; k++) map.push_back(k + l * C.Nx);
    for (int l = 1; l <= C.Nz - 2; l++)
        for (int k = 1; k <= C.Nx - 1; k++) map.push_back((int)C.nu() + k + l * (C.Nx + 1));
    if ((int)map.size() <= MG_DENSE_MAX) {
        C.ndense = (int)map.size();
        size_t n2 = (size_t)C.ndense * C.ndense;
        if (e == cudaSuccess) e = alloc0(&C.dmap, map.size());
        if (e == cudaSuccess) e = cudaMemcpy(C.dmap, map.data(), sizeof(int) * map.size(), cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = alloc0(&C.Awork, n2);
        if (e == cudaSuccess) e = alloc0(&C.AinvT, n2);
    } else {
        for (int q = 0; q < 4; q++) {
            if (e == cudaSuccess) e = alloc0(&C.cg[2 * q], C.nu());
            if (e == cudaSuccess) e = alloc0(&C.cg[2 * q + 1], C.nv());
        }
    }
    if (e != cudaSuccess) return mdz_cuda_check(ctx, e, "multigrid allocation");
    return MDZ_OK;
}

template <typename T>
static void free_hierarchy(mg_hier<T> &H) {
    for (int l = 0; l < H.nlev; l++) {
        mg_level<T> &L = H.L[l];
        if (L.own_tags) { cudaFree(L.BCu); cudaFree(L.BCv); cudaFree(L.BCp); cudaFree(L.BCg); }
        void *p[] = {L.D11, L.D33, L.xu, L.xv, L.yu, L.yv, L.fu, L.fv, L.ru, L.rv, L.idu, L.idv,
                     L.cg[0], L.cg[1], L.cg[2], L.cg[3], L.cg[4], L.cg[5], L.cg[6], L.cg[7],
                     L.dmap, L.Awork, L.AinvT, L.su, L.sv, L.pz};
        for (void *q : p) if (q) cudaFree(q);
    }
    if (H.pmean) cudaFree(H.pmean);
    H.pmean = nullptr;
    H.nlev = 0;
}

template <typename T>
static mdz_status alloc_gcr(mdz_ctx *ctx, gcr_space<T> &S, int m) {
    const mdz_dgrid &g = ctx->g;
    S.nu = (size_t)g.Nx * (g.Nz + 1); S.nv = (size_t)(g.Nx + 1) * g.Nz; S.np = (size_t)g.ncx * g.ncz;
    S.n = S.nu + S.nv + S.np;
    S.ld = (S.n + 31) / 32 * 32;
    S.m = m;
    cudaError_t e = alloc0(&S.Z, S.ld * m);
    if (e == cudaSuccess) e = alloc0(&S.W, S.ld * m);
    T **v[] = {&S.x, &S.r, &S.z, &S.w, &S.t, &S.pin};
    for (T **b : v) if (e == cudaSuccess) e = alloc0(b, S.ld);
    if (e == cudaSuccess) e = cudaMalloc((void **)&S.dA0, sizeof(T *) * (GCR_MAX_M + 4));
    if (e == cudaSuccess) e = alloc0(&S.dots, 4 * (GCR_MAX_M + 8));   // see the layout in gcr_solve
    if (e == cudaSuccess) e = alloc0(&S.tri, (size_t)GCR_MAX_M * GCR_MAX_M + GCR_MAX_M);
    if (e != cudaSuccess) return mdz_cuda_check(ctx, e, "GCR allocation");
    // pointer table: rows 0..m-1 = W_i, row m = w, row m+1 = r
    std::vector<const T *> a0(m + 2);
    for (int i = 0; i < m + 2; i++) a0[i] = i < m ? S.W + S.ld * i : (i == m ? S.w : S.r);
    cudaMemcpy(S.dA0, a0.data(), sizeof(T *) * (m + 2), cudaMemcpyHostToDevice);
    if (sizeof(T) == 4) {
        for (int q = 0; q < 12; q++) {
            size_t n = (q < 8) ? S.np : (size_t)g.Nx * g.Nz;
            if (alloc0(&S.Dc[q], n) != cudaSuccess) return mdz_cuda_check(ctx, cudaGetLastError(), "GCR allocation");
        }
    }
    return MDZ_OK;
}

template <typename T>
static void free_gcr(gcr_space<T> &S) {
    void *p[] = {S.Z, S.W, S.x, S.r, S.z, S.w, S.t, S.pin, S.tri, S.dA0, S.dots};
    for (void *q : p) if (q) cudaFree(q);
    for (int q = 0; q < 12; q++) if (S.Dc[q]) cudaFree(S.Dc[q]);
}

mdz_status mdz_solver_ensure(mdz_ctx *ctx) {
    if (ctx->solver && ctx->solver->ready) return MDZ_OK;
    mdz_status s = mdz_check_stokes_bcs(ctx);
    if (s != MDZ_OK) return s;
    if (!ctx->bcs_box)
        return mdz_fail(ctx, MDZ_ERR_UNSUPPORTED, "solver: boundary tags must be the free-slip box pattern");
    if (!ctx->solver) ctx->solver = new mdz_solver();
    mdz_solver *S = ctx->solver;
    if ((s = build_hierarchy<double>(ctx, S->mg64)) != MDZ_OK) return s;
    if ((s = build_hierarchy<float>(ctx, S->mg32)) != MDZ_OK) return s;
    if ((s = alloc_gcr<double>(ctx, S->g64, S->restart)) != MDZ_OK) return s;
    if ((s = alloc_gcr<float>(ctx, S->g32, S->restart)) != MDZ_OK) return s;
    MDZ_CUDA(ctx, cudaMallocHost((void **)&S->sc, 64 * sizeof(double)));
    memset(S->sc, 0, 64 * sizeof(double));
#define MG_SMEM_ATTR(k, bytes) MDZ_CUDA(ctx, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes))
    MG_SMEM_ATTR((k_galerkin<double, true>), sizeof(double) * MG_NST * GAL_THREADS);
    MG_SMEM_ATTR((k_galerkin<double, false>), sizeof(double) * MG_NST * GAL_THREADS);
    MG_SMEM_ATTR((k_galerkin<float, true>), sizeof(float) * MG_NST * GAL_THREADS);
    MG_SMEM_ATTR((k_galerkin<float, false>), sizeof(float) * MG_NST * GAL_THREADS);
#undef MG_SMEM_ATTR
    S->mg64.bottom = mg_bottom_placed<double>();
    S->mg32.bottom = mg_bottom_placed<float>();
    MDZ_CUDA(ctx, cudaFuncSetAttribute(k_coarse_dense_setup<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       MG_DENSE_SMEM));
    MDZ_CUDA(ctx, cudaFuncSetAttribute(k_coarse_dense_setup<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       MG_DENSE_SMEM));
    MDZ_CUDA(ctx, cudaDeviceSynchronize());
    S->ready = true;
    return MDZ_OK;
}

template <typename T>
static mdz_status copy_stencils(mdz_ctx *ctx, mg_hier<T> &H, int level, int *Nx, int *Nz, double *su,
                                double *sv) {
    if (level < 0 || level >= H.nlev) return mdz_fail(ctx, MDZ_ERR_ARG, "mg_stencils: level %d of %d", level, H.nlev);
    const mg_level<T> &L = H.L[level];
    *Nx = L.Nx;
    *Nz = L.Nz;
    if (level == 0 && H.viscous && (su || sv)) {   // the viscous level keeps no stencils of its own
        k_picard_stencil<T><<<dim3((L.Nx + 32) / 32, (L.Nz + 8) / 8), dim3(32, 8), 0, ctx->stream>>>(
            H.setup_geom, L.D11, L.D33, L.su, L.sv);
        MDZ_LAUNCHED(ctx);
    }
    MDZ_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    const T *src[2] = {L.su, L.sv};
    double *dst[2] = {su, sv};
    size_t cnt[2] = {MG_NST * L.nu(), MG_NST * L.nv()};
    for (int q = 0; q < 2; q++) {
        if (!dst[q]) continue;
        std::vector<T> h(cnt[q]);
        MDZ_CUDA(ctx, cudaMemcpy(h.data(), src[q], sizeof(T) * cnt[q], cudaMemcpyDeviceToHost));
        for (size_t i = 0; i < cnt[q]; i++) dst[q][i] = (double)h[i];
    }
    return MDZ_OK;
}

extern "C" mdz_status mdz_mg_stencils(mdz_ctx *ctx, int precision, int level, int *levels, int *Nx, int *Nz,
                                      double *su, double *sv) {
    if (!ctx || !Nx || !Nz || !levels) return ctx ? mdz_fail(ctx, MDZ_ERR_ARG, "mg_stencils: null argument") : MDZ_ERR_ARG;
    if (!ctx->solver || !ctx->solver->ready)
        return mdz_fail(ctx, MDZ_ERR_STATE, "mg_stencils: no multigrid hierarchy (run a solve first)");
    if (precision == 64) {
        *levels = ctx->solver->mg64.nlev;
        return copy_stencils<double>(ctx, ctx->solver->mg64, level, Nx, Nz, su, sv);
    }
    if (precision == 32) {
        *levels = ctx->solver->mg32.nlev;
        return copy_stencils<float>(ctx, ctx->solver->mg32, level, Nx, Nz, su, sv);
    }
    return mdz_fail(ctx, MDZ_ERR_ARG, "mg_stencils: precision 64 or 32");
}

extern "C" mdz_status mdz_set_solver_options(mdz_ctx *ctx, int nu1, int nu2, double omega, int restart, int check,
                                             int mg_jacobian) {
    if (!ctx) return MDZ_ERR_ARG;
    if (nu1 < 1 || nu1 > 16 || nu2 < 0 || nu2 > 16 || !(omega > 0.0 && omega < 2.0) || restart < 2 ||
        restart > GCR_MAX_M || check < 1 || check > 64 || (mg_jacobian != 0 && mg_jacobian != 1))
        return mdz_fail(ctx, MDZ_ERR_ARG, "solver options: nu1 1..16, nu2 0..16, omega in (0, 2), restart 2..%d, "
                                          "check 1..64, mg_jacobian 0/1", GCR_MAX_M);
    if (!ctx->solver) ctx->solver = new mdz_solver();
    mdz_solver *S = ctx->solver;
    MDZ_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    for (int q = 0; q < MDZ_PRE_SLOTS; q++)
        if (S->pre[q]) { cudaGraphExecDestroy(S->pre[q]); S->pre[q] = nullptr; }
    S->nu1 = nu1; S->nu2 = nu2; S->omega = omega; S->check = check; S->mg_jacobian = mg_jacobian;
    if (S->ready && restart != S->restart) {
        free_gcr(S->g64);
        free_gcr(S->g32);
        S->g64 = gcr_space<double>();
        S->g32 = gcr_space<float>();
        S->restart = restart;
        mdz_status s;
        if ((s = alloc_gcr<double>(ctx, S->g64, restart)) != MDZ_OK) return s;
        if ((s = alloc_gcr<float>(ctx, S->g32, restart)) != MDZ_OK) return s;
    }
    S->restart = restart;
    return MDZ_OK;
}

extern "C" mdz_status mdz_set_schur_scaling(mdz_ctx *ctx, int mode) {
    if (!ctx) return MDZ_ERR_ARG;
    if (mode != 0 && mode != 1) return mdz_fail(ctx, MDZ_ERR_ARG, "Schur scaling: mode 0 or 1");
    if (!ctx->solver) ctx->solver = new mdz_solver();
    ctx->solver->schur = mode;   // graphs of both kinds have their own slots
    return MDZ_OK;
}

// The grid spacing changed (PureShearALE): every level's spacing follows the
// fine one (doubling per level, as the hierarchy was built) and the captured
// preconditioner graphs, which hold the old spacings as kernel arguments, are
// dropped (recaptured on their next use).
mdz_status mdz_solver_regrid(mdz_ctx *ctx) {
    mdz_solver *S = ctx->solver;
    if (!S) return MDZ_OK;
    MDZ_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    for (int q = 0; q < MDZ_PRE_SLOTS; q++)
        if (S->pre[q]) { cudaGraphExecDestroy(S->pre[q]); S->pre[q] = nullptr; S->pre_eta[q] = nullptr; }
    S->mg64.built = false;   // no solve may keep operators of the old spacing
    S->mg32.built = false;
    double dx = ctx->g.dx, dz = ctx->g.dz;
    for (int lev = 0; lev < S->mg64.nlev; lev++, dx *= 2, dz *= 2) { S->mg64.L[lev].dx = dx; S->mg64.L[lev].dz = dz; }
    dx = ctx->g.dx; dz = ctx->g.dz;
    for (int lev = 0; lev < S->mg32.nlev; lev++, dx *= 2, dz *= 2) { S->mg32.L[lev].dx = dx; S->mg32.L[lev].dz = dz; }
    return MDZ_OK;
}

void mdz_solver_free(mdz_ctx *ctx) {
    if (!ctx->solver) return;
    mdz_solver *S = ctx->solver;
    for (int q = 0; q < MDZ_PRE_SLOTS; q++)
        if (S->pre[q]) cudaGraphExecDestroy(S->pre[q]);
    free_hierarchy(S->mg64);
    free_hierarchy(S->mg32);
    free_gcr(S->g64);
    free_gcr(S->g32);
    if (S->sc) cudaFreeHost(S->sc);
    delete S;
    ctx->solver = nullptr;
}

int mdz_solver_levels(const mdz_ctx *ctx) { return ctx->solver ? ctx->solver->mg64.nlev : 0; }

// ---------------------------------------------------------------------------
// Multigrid setup (coefficients) and V-cycle.
template <typename T>
static mdz_status mg_setup(mdz_ctx *ctx, mg_hier<T> &H, const double *eta_n, const double *eta_s,
                           const stokes_coefs<T> &K, bool newton, cudaStream_t st) {
    mg_level<T> &F = H.L[0];
    int nc = F.ncx * F.ncz, nv = F.Nx * F.Nz;
    H.newton = newton;
    H.built = true;
    H.viscous = !newton;
    H.setup_geom = F.geom();
    cudaEvent_t ev;
    mdz_prof_begin(ctx, MDZ_PROF_MG_SETUP, st, &ev);
    k_fill_D11_D33<T><<<mdz_blocks(nv > nc ? nv : nc), MDZ_THREADS, 0, st>>>(nc, nv, eta_n, eta_s, F.D11, F.D33);
    MDZ_LAUNCHED(ctx);
    // level-0 stencils: the Picard block written out from eta, or the Newton
    // Jacobian's velocity block probed with 2 x 16 colour classes
    const dim3 bl(32, 8), gr0((F.Nx + 1 + 31) / 32, (F.Nz + 1 + 7) / 8);
    if (!newton) {   // (stored only where something reads them: mdz_mg_stencils writes them out on request)
        if (H.nlev == 1) {
            k_picard_stencil<T><<<gr0, bl, 0, st>>>(F.geom(), F.D11, F.D33, F.su, F.sv);
            MDZ_LAUNCHED(ctx);
        }
    } else {
        MDZ_CUDA(ctx, cudaMemsetAsync(F.su, 0, sizeof(T) * MG_NST * F.nu(), st));
        MDZ_CUDA(ctx, cudaMemsetAsync(F.sv, 0, sizeof(T) * MG_NST * F.nv(), st));
        for (int comp = 0; comp < 2; comp++)
            for (int cz = 0; cz < MG_PROBE; cz++)
                for (int cx = 0; cx < MG_PROBE; cx++) {
                    k_probe_vec<T><<<gr0, bl, 0, st>>>(F.geom(), comp, cx, cz, F.xu, F.xv);
                    MDZ_LAUNCHED(ctx);
                    k_mg_apply<T><<<gr0, bl, 0, st>>>(F.geom(), K, F.xu, F.xv, F.pz, F.ru, F.rv);
                    MDZ_LAUNCHED(ctx);
                    k_probe_collect<T><<<gr0, bl, 0, st>>>(F.geom(), comp, cx, cz, F.ru, F.rv, F.su, F.sv);
                    MDZ_LAUNCHED(ctx);
                }
    }
    {   // Jacobi diagonal of level 0: the viscosity formula (Picard) or the probed stencil (Newton)
        size_t n = F.nu() > F.nv() ? F.nu() : F.nv();
        if (newton) k_st_diag<T><<<mdz_blocks(n), MDZ_THREADS, 0, st>>>(F.geom(), F.su, F.sv, F.idu, F.idv);
        else k_mg_diag<T><<<mdz_blocks(n), MDZ_THREADS, 0, st>>>(F.geom(), F.D11, F.D33, F.idu, F.idv);
        MDZ_LAUNCHED(ctx);
    }
    int *status = ctx->d_counters + 40;   // [0] coarse inverse, [1] Galerkin footprint
    MDZ_CUDA(ctx, cudaMemsetAsync(status, 0, 2 * sizeof(int), st));
    for (int l = 1; l < H.nlev; l++) {
        mg_level<T> &P = H.L[l - 1], &L = H.L[l];
        const int ub = (int)((L.nu() + 31) / 32), vb = (int)((L.nv() + 31) / 32);
        const size_t smem = sizeof(T) * MG_NST * GAL_THREADS;
        if (l == 1 && !newton)
            MDZ_PDL(ctx, k_galerkin<T, true>, ub + vb, GAL_THREADS, smem, st, P.geom(), nullptr, nullptr, P.D11, P.D33,
                    L.geom(), ub, L.su, L.sv, L.idu, L.idv, status + 1);
        else
            MDZ_PDL(ctx, k_galerkin<T, false>, ub + vb, GAL_THREADS, smem, st, P.geom(), P.su, P.sv, nullptr, nullptr,
                    L.geom(), ub, L.su, L.sv, L.idu, L.idv, status + 1);
    }
    mg_level<T> &C = H.L[H.nlev - 1];
    if (C.ndense) {
        const size_t smem = (size_t)C.ndense * C.ndense * sizeof(T);
        k_coarse_dense_setup<T><<<1, 512, smem <= MG_DENSE_SMEM ? smem : 0, st>>>(C.geom(), C.su, C.sv, C.ndense,
                                                                              C.dmap, C.Awork, C.AinvT, status);
        MDZ_LAUNCHED(ctx);
    }
    {   // algorithmic bytes: viscosities in, D11 / D33 out; each Galerkin level
        // reads the finer stencils (the first one the viscosities) once and
        // writes its own plus the inverse diagonal
        double b = 8.0 * (nc + nv) + 2.0 * sizeof(T) * (nc + nv);
        for (int l = 1; l < H.nlev; l++)
            b += sizeof(T) * ((l > 1 || newton ? MG_NST : 0.0) * (double)(H.L[l - 1].nu() + H.L[l - 1].nv()) +
                              (MG_NST + 1.0) * (double)(H.L[l].nu() + H.L[l].nv()));
        mdz_prof_end(ctx, MDZ_PROF_MG_SETUP, b, st, ev);
    }
    MDZ_CUDA(ctx, cudaMemcpyAsync((int *)(ctx->solver->sc + 20), status, 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
    return MDZ_OK;
}

static inline dim3 box_grid(int Nx, int Nz) { return dim3((Nx + 1 + 31) / 32, (Nz + 1 + 7) / 8); }

// Whether the FP64 level-0 kernels of a grid take tiles of 16 x 4 points and the
// restriction tiles of 8 x 4 coarse points: where the 32 x 8 (16 x 8) tiles leave
// SMs idle, or little more than one to each.  A warp's FP64 instruction takes its
// scheduler's unit 64 clocks, so eight warps on one SM in three take three times
// as long as spread out.  V-cycle, before and after: 100 x 100 cells 72.9 and
// 68.4 us, 120 x 60 62.6 and 58.2, 256 x 128 (153 tiles) 78.3 and 76.0; from
// 200 tiles on (400 x 400: 181 and 181) the smaller halo of the large tiles
// counts.  FP32 is not bound by that unit.
#define MG_SMALL_W 16
#define MG_SMALL_H 4
#define MG_SMALL_TILES 200
#define MG_RR_W 8
#define MG_RR_H 4
#define MG_RR_T 352
#define MG_RR_TILES 152
template <typename T>
static bool mg_small_tiles(int Nx, int Nz) {
    return sizeof(T) == 8 && ((Nx + 32) / 32) * ((Nz + 8) / 8) < MG_SMALL_TILES;
}
template <typename T>
static bool mg_small_coarse(int Nxc, int Nzc) {
    return sizeof(T) == 8 && ((Nxc + 16) / 16) * ((Nzc + 8) / 8) < MG_RR_TILES;
}

// Shared memory per CTA of the bottom kernel run from level l down.
template <typename T>
static size_t mg_bottom_bytes(const mg_hier<T> &H, int l) {
    long long n = 0;
    for (int q = l; q < H.nlev - 1; q++) n += mg_bottom_level_elems(H.L[q].Nx, H.L[q].Nz);
    const mg_level<T> &C = H.L[H.nlev - 1];
    n += mg_bottom_box(C.Nx, C.Nz) + (long long)C.ndense * (1 + mg_bottom_share(C.ndense));
    return (size_t)n * sizeof(T);
}

// Whether vcycle() runs level l and all below it in the one-launch bottom
// kernel: as soon as their data fit the cluster's shared memory and the level
// has at most 2048 rows in FP64 (33 x 32 cells), 4096 in FP32 (64 x 32 and a
// little).  V-cycle of 100 x 100, 256 x 128 and 400 x 400 cells in FP64, us:
//   limit   256     600     2048
//           85      77      73
//           89      84      80
//           199     188     184
#define MG_BOTTOM_ROWS64 2048
#define MG_BOTTOM_ROWS32 4096
template <typename T>
static bool vcycle_bottom(const mg_hier<T> &H, int l) {
    const mg_level<T> &L = H.L[l];
    const bool viscous = l == 0 && !H.newton;   // level 0 of a Picard hierarchy: stencil from eta directly
    return H.bottom && !viscous && l < H.nlev - 1 && H.L[H.nlev - 1].ndense && H.nlev - l <= MG_BOTTOM_MAX &&
           mg_bottom_rows(L.Nx, L.Nz) <= (sizeof(T) == 4 ? MG_BOTTOM_ROWS32 : MG_BOTTOM_ROWS64) &&
           mg_bottom_bytes<T>(H, l) <= MG_BOTTOM_SMEM;
}

// Whether vcycle() smooths level l with its own sweeps (not the dense
// coarsest solve, the coarse CG, nor the one-launch bottom kernel).
template <typename T>
static bool vcycle_smoothed(const mg_hier<T> &H, int l) {
    return l < H.nlev - 1 && !vcycle_bottom<T>(H, l);
}

// One V-cycle: H.L[l].x <- approx A^-1 H.L[l].f.  Level 0 smooths with the
// re-discretised stencil (viscosities read directly), coarser levels with the
// Galerkin stencils.  x0_done: the first sweep from x = 0 (x = omega D^-1 f)
// was already written into L.xu / L.xv with the right-hand side (by
// k_precond, or by the finer level's restriction); out_u / out_v: where
// the last post-smoothing sweep writes (the caller's vector), else the level's
// own buffers.  Both only for a level that vcycle_smoothed() accepts.  zp: the
// pressure to shift by its mean in the last launch (viscous level 0, nu2 = 1).
template <typename T>
static mdz_status vcycle(mdz_ctx *ctx, mg_hier<T> &H, int l, int nu1, int nu2, T omega, cudaStream_t st,
                         bool x0_done = false, T *out_u = nullptr, T *out_v = nullptr, T *zp = nullptr) {
    mg_level<T> &L = H.L[l];
    stokes_geom G = L.geom();
    stokes_coefs<T> D = L.coefs();
    const dim3 bl(32, 8), gr = box_grid(L.Nx, L.Nz);
    // (const views: launch_pdl converts its arguments to the kernel's types)
    if (l == H.nlev - 1 && L.ndense) {
        MDZ_PDL(ctx, k_coarse_dense_solve<T>, 1, 512, 0, st, L.ndense, (int)L.nu(), (int)L.nv(), L.dmap, L.AinvT,
                L.fu, L.fv, L.xu, L.xv);
        return MDZ_OK;
    }
    if (l == H.nlev - 1) {
        int maxit = 4 * (L.ncx > L.ncz ? L.ncx : L.ncz) + 50;
        k_mg_coarse_cg<T><<<1, 1024, 0, st>>>(G, L.su, L.sv, L.fu, L.fv, L.idu, L.idv, L.xu, L.xv, L.ru, L.rv,
                                              L.cg[0], L.cg[1], L.cg[2], L.cg[3], L.cg[4], L.cg[5], maxit, 1e-6);
        MDZ_LAUNCHED(ctx);
        return MDZ_OK;
    }
    const bool viscous = l == 0 && !H.newton;   // level 0 of a Picard hierarchy: stencil from eta directly
    if (vcycle_bottom<T>(H, l)) {   // this level and all below in one launch
        const mg_level<T> &Cd = H.L[H.nlev - 1];
        mg_bottom_args<T> A;
        A.nlev = H.nlev - l; A.nu1 = nu1; A.nu2 = nu2; A.ndense = Cd.ndense; A.omega = omega;
        A.dmap = Cd.dmap; A.AinvT = Cd.AinvT;
        for (int q = 0; q < A.nlev; q++) {
            const mg_level<T> &B = H.L[l + q];
            A.Nx[q] = B.Nx; A.Nz[q] = B.Nz;
            A.su[q] = B.su; A.sv[q] = B.sv; A.idu[q] = B.idu; A.idv[q] = B.idv;
        }
        A.fu = L.fu; A.fv = L.fv; A.xu = L.xu; A.xv = L.xv;
        MDZ_PDL_CLUSTER(ctx, MG_BOTTOM_CTAS, k_mg_bottom<T>, MG_BOTTOM_CTAS, mg_bottom_threads<T>(), mg_bottom_bytes<T>(H, l), st, A);
        return MDZ_OK;
    }
    const int rows_grid = mdz_blocks(L.nu() + L.nv(), ST_THREADS);
    const bool small = mg_small_tiles<T>(L.Nx, L.Nz);
    auto tiles = [&](int w, int h) { return dim3((L.Nx + w) / w, (L.Nz + h) / h); };
    auto smooth = [&](const T *xu, const T *xv, T *ou, T *ov) -> mdz_status {
        if (viscous && small)
            MDZ_PDL(ctx, (k_mg_smooth<T, MG_SMALL_W, MG_SMALL_H>), tiles(MG_SMALL_W, MG_SMALL_H), MG_SMALL_W * MG_SMALL_H, 0,
                    st, G, D, xu, xv, L.fu, L.fv, L.idu, L.idv, omega, ou, ov);
        else if (viscous)
            MDZ_PDL(ctx, (k_mg_smooth<T, 32, 8>), gr, 256, 0, st, G, D, xu, xv, L.fu, L.fv, L.idu, L.idv, omega, ou, ov);
        else MDZ_PDL(ctx, k_st_smooth<T>, rows_grid, ST_THREADS, 0, st, G, L.su, L.sv, xu, xv, L.fu, L.fv, L.idu, L.idv,
                     omega, ou, ov);
        return MDZ_OK;
    };
    mdz_status s;
    // pre-smoothing from x = 0
    if (!x0_done && (s = smooth(nullptr, nullptr, L.xu, L.xv)) != MDZ_OK) return s;
    for (int q = 1; q < nu1; q++) {
        if ((s = smooth(L.xu, L.xv, L.yu, L.yv)) != MDZ_OK) return s;
        std::swap(L.xu, L.yu); std::swap(L.xv, L.yv);
    }
    // residual, restriction and the coarse level's first sweep in one launch
    mg_level<T> &C = H.L[l + 1];
    const stokes_geom GC = C.geom();
    const bool c0 = vcycle_smoothed<T>(H, l + 1);
    T *cxu = c0 ? C.xu : nullptr, *cxv = c0 ? C.xv : nullptr;
    const int cw = C.Nx + 1, ch = C.Nz + 1;
    const long long cpts = (long long)cw * ch;
#define MG_RR(kernel, TX, TY, NT, ...)                                                                                \
    MDZ_PDL(ctx, kernel<T, TX, TY, NT>, dim3((cw + TX - 1) / TX, (ch + TY - 1) / TY), NT, 0, st, G, __VA_ARGS__, L.xu, \
            L.xv, L.fu, L.fv, GC, C.fu, C.fv, C.idu, C.idv, omega, cxu, cxv)
    if (viscous && mg_small_coarse<T>(C.Nx, C.Nz)) MG_RR(k_mg_resid_restrict, MG_RR_W, MG_RR_H, MG_RR_T, D);
    else if (viscous) MG_RR(k_mg_resid_restrict, 16, 8, 384, D);
    else if (cpts > MG_TILE_LARGE) MG_RR(k_st_resid_restrict, 16, 8, 416, L.su, L.sv);
    else if (cpts > MG_TILE_SMALL) MG_RR(k_st_resid_restrict, 8, 4, 352, L.su, L.sv);
    else MG_RR(k_st_resid_restrict, 4, 2, 128, L.su, L.sv);
#undef MG_RR
    if ((s = vcycle<T>(ctx, H, l + 1, nu1, nu2, omega, st, c0)) != MDZ_OK) return s;
    if (nu2 == 0) {
        MDZ_PDL(ctx, k_mg_prolong_add<T>, gr, bl, 0, st, G, GC, C.xu, C.xv, L.xu, L.xv);
        return MDZ_OK;
    }
    // prolongation and the first post-smoothing sweep in one launch; the last
    // sweep goes straight into the caller's vector
    T *ou = nu2 == 1 && out_u ? out_u : L.yu, *ov = nu2 == 1 && out_u ? out_v : L.yv;
    if (viscous && small)
        MDZ_PDL(ctx, (k_mg_prolong_smooth<T, MG_SMALL_W, MG_SMALL_H>), tiles(MG_SMALL_W, MG_SMALL_H),
                MG_SMALL_W * MG_SMALL_H, 0, st, G, D, GC, C.xu, C.xv, L.xu, L.xv, L.fu, L.fv, L.idu, L.idv, omega, ou, ov,
                zp, H.pmean);
    else if (viscous)
        MDZ_PDL(ctx, k_mg_prolong_smooth<T, 32, 8>, gr, 256, 0, st, G, D, GC, C.xu, C.xv, L.xu, L.xv, L.fu, L.fv, L.idu,
                L.idv, omega, ou, ov, zp, H.pmean);
    else if ((long long)(L.Nx + 1) * (L.Nz + 1) > MG_TILE_SMALL)
        MDZ_PDL(ctx, k_st_prolong_smooth<T, 16, 8>, dim3((L.Nx + 16) / 16, (L.Nz + 8) / 8), 256, 0, st, G, GC, L.su, L.sv,
                C.xu, C.xv, L.xu, L.xv, L.fu, L.fv, L.idu, L.idv, omega, ou, ov);
    else
        MDZ_PDL(ctx, k_st_prolong_smooth<T, 8, 4>, dim3((L.Nx + 8) / 8, (L.Nz + 4) / 4), 64, 0, st, G, GC, L.su, L.sv,
                C.xu, C.xv, L.xu, L.xv, L.fu, L.fv, L.idu, L.idv, omega, ou, ov);
    if (ou == L.yu) { std::swap(L.xu, L.yu); std::swap(L.xv, L.yv); }
    for (int q = 1; q < nu2; q++) {
        if (q == nu2 - 1 && out_u) return smooth(L.xu, L.xv, out_u, out_v);
        if ((s = smooth(L.xu, L.xv, L.yu, L.yv)) != MDZ_OK) return s;
        std::swap(L.xu, L.yu); std::swap(L.xv, L.yv);
    }
    return MDZ_OK;
}

// ---------------------------------------------------------------------------
// Pressure mean over the pressure equations (sum, count) and its removal.
// (sum in the vector's precision and an integer count per thread, warp sums
// in that precision, then a fixed-order FP64 sum of the block partials:
// reduce.cuh)
template <typename T>
__global__ void __launch_bounds__(256) k_psum(int np, const signed char *__restrict__ tp, const T *__restrict__ p,
                                              double *part, unsigned int *counter, double *out) {
    T acc = 0;
    int cnt = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < np; i += gridDim.x * blockDim.x)
        if (tp[i] == -1) { acc += p[i]; cnt++; }
    const T v[2] = {acc, (T)cnt};   // (counts per thread are small integers: exact in T)
    mdz_grid_sum<2, T>(v, part, counter, out);
}

// (the mean in the vector's precision: an FP64 division per thread is a long
// instruction sequence on this part)
template <typename T>
__global__ void k_psub(int np, const signed char *__restrict__ tp, const double *__restrict__ sum, T *__restrict__ p) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < np && tp[i] == -1 && sum[1] > 0) p[i] -= (T)sum[0] / (T)sum[1];
}

// ---------------------------------------------------------------------------
// Block preconditioner: zp = (eta_n / celvol) rp ; zu = V-cycle(ru - B zp).
// One launch writes zp (eta_n / celvol from the level-0 copy D11 = 2 eta_n in
// precision T, or from the Jacobian's tangent D11 where that is positive),
// f = r_vel - B zp on the fine level (B: celvol-scaled pressure gradient), with xu non-null the V-cycle's first
// sweep from x = 0, x = omega D^-1 f, and the sum, count and mean of zp over the
// pressure equations for the zero-mean projection in the last launch.
template <typename T, int TW, int TH>
__global__ void __launch_bounds__(TW *TH) k_precond(stokes_geom G, const T *__restrict__ D11, const T *__restrict__ Dt,
                                                 const T *__restrict__ ru, const T *__restrict__ rv,
                                                 const T *__restrict__ rp, T *__restrict__ zp, T *__restrict__ fu,
                                                 T *__restrict__ fv, const T *__restrict__ idu,
                                                 const T *__restrict__ idv, T omega, T *__restrict__ xu,
                                                 T *__restrict__ xv, double *part, unsigned int *counter,
                                                 double *psum) {
    mg_release<T>();
    __shared__ T s_z[TH + 1][TW + 1];   // zp of the centroids from (i0 - 1, j0 - 1)
    const int Nx = G.Nx, Nz = G.Nz, ncx = G.ncx, ncz = G.ncz, a = threadIdx.x % TW, h = threadIdx.x / TW;
    const int ntx = (Nx + TW) / TW, ntiles = ntx * ((Nz + TH) / TH);
    const T half_ivol = T(0.5) * gc<T>(G, GC_IXZ);
    T acc = 0;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int i0 = (tile % ntx) * TW, j0 = (tile / ntx) * TH, i = i0 + a, j = j0 + h;
        for (int t = threadIdx.x; t < (TW + 1) * (TH + 1); t += TW * TH) {
            const int k = i0 - 1 + t % (TW + 1), l = j0 - 1 + t / (TW + 1);
            T v = 0;
            if (k >= 0 && k < ncx && l >= 0 && l < ncz) {
                const int c = k + l * ncx;
                T d = D11[c];
                if (Dt) {   // the Jacobian's tangent D11 where it is positive
                    const T dt = Dt[c];
                    if (dt > T(0)) d = dt;
                }
                v = half_ivol * d * rp[c];
            }
            s_z[t / (TW + 1)][t % (TW + 1)] = v;
        }
        __syncthreads();
        if (i < Nx && j <= Nz) {
            const int c = i + j * Nx;
            T r = 0, x0 = 0;
            if (u_unknown(i, j, Nx, Nz)) {
                r = ru[c] - gc<T>(G, GC_DZ) * (s_z[h][a + 1] - s_z[h][a]);
                if (xu) x0 = omega * idu[c] * r;
            }
            fu[c] = r;
            if (xu) xu[c] = x0;
        }
        if (i <= Nx && j < Nz) {
            const int c = i + j * (Nx + 1);
            T r = 0, x0 = 0;
            if (v_unknown(i, j, Nx, Nz)) {
                r = rv[c] - gc<T>(G, GC_DX) * (s_z[h + 1][a] - s_z[h][a]);
                if (xv) x0 = omega * idv[c] * r;
            }
            fv[c] = r;
            if (xv) xv[c] = x0;
        }
        if (i < ncx && j < ncz) {
            const T v = s_z[h + 1][a + 1];
            zp[i + j * ncx] = v;
            acc += v;
        }
        __syncthreads();
    }
    const T v[1] = {acc};
    if (mdz_grid_sum<1, T>(v, part, counter, psum)) {
        __syncthreads();
        if (threadIdx.x == 0) psum[2] = (double)((T)psum[0] / (T)(ncx * ncz));
    }
}

// z pressure <- zero mean over the pressure equations (the mean cancels in
// the gradient of the right-hand side, so it is removed only here)
template <typename T>
__global__ void k_pmean_out(int np, const double *psum, T *zp) {
    mg_release<T>();
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < np) zp[i] -= (T)psum[2];
}

// z velocity <- the V-cycle's result; z pressure <- zero mean, as k_pmean_out
template <typename T>
__global__ void k_copy_out(size_t nu, size_t nv, int np, const T *xu, const T *xv, const double *psum,
                           T *__restrict__ zu, T *__restrict__ zv, T *zp) {
    mg_release<T>();
    pdl_wait();
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nu) zu[i] = xu[i];
    if (i < nv) zv[i] = xv[i];
    if (i < (size_t)np) zp[i] -= (T)psum[2];
}

// (captured: the first launch must be an ordinary one, so that the graph as a
// whole follows the stream's earlier work)
template <typename T>
static mdz_status precondition(mdz_ctx *ctx, mg_hier<T> &H, const T *Dt, const T *r, T *z, size_t nu, size_t nv,
                               cudaStream_t st) {
    mg_level<T> &F = H.L[0];
    stokes_geom G = F.geom();
    const int np = F.ncx * F.ncz;
    mdz_solver *S = ctx->solver;
    // a level-0 V-cycle of its own sweeps takes its first sweep from the
    // right-hand side kernel and writes its last sweep into z
    const bool fused = vcycle_smoothed<T>(H, 0) && S->nu2 > 0;
    const bool mean_fused = fused && !H.newton && S->nu2 == 1;
    T *const zp = z + nu + nv;
    // zero-mean pressure block: constants are the operator's null space; left
    // in, they grow in the iterates and cost the FP32 gradients their accuracy
    const bool small = mg_small_tiles<T>(F.Nx, F.Nz);
    const int tw = small ? MG_SMALL_W : 32, th = small ? MG_SMALL_H : 8;
    int blocks = ((F.Nx + tw) / tw) * ((F.Nz + th) / th);
    if (blocks > 152 * 8) blocks = 152 * 8;
#define PRECOND(W, H_)                                                                                                   \
    k_precond<T, W, H_><<<blocks, W * H_, 0, st>>>(G, F.D11, Dt, r, r + nu, r + nu + nv, zp, F.fu, F.fv, F.idu, F.idv,   \
                                                   (T)S->omega, fused ? F.xu : nullptr, fused ? F.xv : nullptr,          \
                                                   ctx->red_part + MDZ_RP_PRECP, ctx->red_cnt + MDZ_RC_PRECP, H.pmean)
    if (small) PRECOND(MG_SMALL_W, MG_SMALL_H);
    else PRECOND(32, 8);
#undef PRECOND
    MDZ_LAUNCHED(ctx);
    mdz_status s = vcycle<T>(ctx, H, 0, S->nu1, S->nu2, (T)S->omega, st, fused, fused ? z : nullptr,
                             fused ? z + nu : nullptr, mean_fused ? zp : nullptr);
    if (s != MDZ_OK || mean_fused) return s;
    if (fused) {
        MDZ_PDL(ctx, k_pmean_out<T>, mdz_blocks(np), MDZ_THREADS, 0, st, np, H.pmean, zp);
    } else {
        size_t n = nu > nv ? nu : nv;
        if ((size_t)np > n) n = np;
        MDZ_PDL(ctx, k_copy_out<T>, mdz_blocks(n), MDZ_THREADS, 0, st, nu, nv, np, F.xu, F.xv, H.pmean, z, z + nu, zp);
    }
    return MDZ_OK;
}

// ---------------------------------------------------------------------------
// GCR kernels (vectors are u|v|p contiguous of length n).
// Orthogonalisation: classical Gram-Schmidt, with a second pass only where
// the first removed all but 1e-3 (FP64 basis) or 1e-1 (FP32 basis) of w's
// squared norm (a DGKS-type test; with the usual 1/2 the second pass ran in
// almost every FP32 iteration and made the plain FP64 solve 7 % slower for
// the same iteration counts; 1e-3 on FP32 bases cost 15-25 % more iterations
// on a 401^2 visco-elasto-plastic box),
// decided on the device: the first pass's k_gcr_dots sets sc[5] = 1 for a
// second pass, and the second-pass kernels return at once when it is 0.
// dots[0..k-1] = (w, W_q), dots[k] = (w, w), dots[k+1] = (w, r) of the pass
// whose coefficients the finish applies; sc[0] = 1/||w||, sc[1] = alpha,
// sc[2] = ||w||^2, sc[3] = running ||r||^2 (so the host reads it only every
// few iterations).
// The running norm also goes to the host's memory with the iteration's ticket:
// the host decides on the next iteration while the finish is still running,
// instead of copying sc[3] back after it.
// One warp: lane q holds d[q], d[q + 32], and dd is sum d^2; wa becomes
// sum d alpha.  (One thread took two chains of k dependent FP64
// instructions; with the folded block sums a launch went from 8.2 .. 12.4 us to
// 7.2 .. 8.3, for 1 .. 30 vectors of 30 000.)
__device__ __forceinline__ void gcr_scalars(int k, const double *d, double dk, double dr, double dd, double *sc, double *tri,
                                            bool second, volatile double *note, double ticket) {
    // column k of U: the pass's Gram-Schmidt coefficients (added to the first
    // pass's after a second pass) and the new direction's norm
    double *U = tri + (size_t)k * GCR_MAX_M;
    double wa = 0.0;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int q = 32 * h + (threadIdx.x & 31);
        if (q < k) {
            wa += d[h] * sc[8 + q];
            U[q] = second ? U[q] + d[h] : d[h];
        }
    }
    wa = warp_sum_all(wa);
    if ((threadIdx.x & 31) != 0) return;
    const double nrm2 = dk - dd, wr = dr - wa;   // (w - sum beta_q W_q, r0) = (w, r0) - sum beta_q alpha_q
    double nrm = sqrt(nrm2 > 0 ? nrm2 : 0.0);
    const double inrm = nrm > 0 ? 1.0 / nrm : 0.0;
    double alpha = nrm > 0 ? wr / nrm : 0.0;   // alpha_k = (W_k, r0) = (W_k, r_k): W orthonormal
    U[k] = nrm;
    sc[0] = inrm;
    sc[1] = alpha;
    sc[2] = nrm2;
    const double rr = sc[3] - alpha * alpha;   // ||r_k||^2 = ||r_k-1||^2 - alpha_k^2
    sc[3] = rr;
    sc[8 + k] = alpha;
    note[0] = rr;
    __threadfence_system();
    note[1] = ticket;
}

// gamma = U^-1 alpha: x = x0 + Z gamma with the raw preconditioned vectors Z,
// whose orthogonalised combinations Z U^-1 are the directions whose images are
// the orthonormal W.  Back substitution by one warp, a column at a time: lane i
// keeps rows i and i + 32, quotients by the reciprocal of the diagonal with one
// step on the remainder (Markstein, IBM J. Res. Dev. 34, 1990).  One thread, row
// by row, took 33 us for 30 columns, this 9.
__global__ void __launch_bounds__(32) k_gcr_gamma(int k, const double *__restrict__ sc, double *__restrict__ tri) {
    double *g = tri + (size_t)GCR_MAX_M * GCR_MAX_M;
    const int lane = threadIdx.x;
    double v[2], dg[2], rd[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int i = 32 * h + lane;
        v[h] = i < k ? sc[8 + i] : 0.0;
        dg[h] = i < k ? tri[(size_t)i * GCR_MAX_M + i] : 0.0;
        rd[h] = fabs(dg[h]) >= 2.2250738585072014e-308 ? 1.0 / dg[h] : 0.0;   // (no subnormal: 1 / dg overflows)
    }
    double gv[2] = {0.0, 0.0};
    auto column = [&](int j, double &u0, double &u1) {   // rows above the diagonal
        const double *U = tri + (size_t)j * GCR_MAX_M;
        u0 = lane < j ? U[lane] : 0.0;
        u1 = 32 + lane < j ? U[32 + lane] : 0.0;
    };
    double u0, u1, n0 = 0.0, n1 = 0.0;   // this column and the next
    column(k - 1, u0, u1);
    for (int j = k - 1; j >= 0; j--) {
        if (j > 0) column(j - 1, n0, n1);
        const bool hi = j >= 32;
        const double vj = hi ? v[1] : v[0], dj = hi ? dg[1] : dg[0], rj = hi ? rd[1] : rd[0];
        double q = vj * rj;
        q = __fma_rn(__fma_rn(-q, dj, vj), rj, q);
        q = __shfl_sync(0xffffffffu, q, j & 31);
        if (lane == (j & 31)) { if (hi) gv[1] = q; else gv[0] = q; }
        v[0] -= u0 * q;
        v[1] -= u1 * q;
        u0 = n0;
        u1 = n1;
    }
#pragma unroll
    for (int h = 0; h < 2; h++)
        if (32 * h + lane < k) g[32 * h + lane] = gv[h];
}

__global__ void k_set_scalar(double *dst, const double *src) {
    if (threadIdx.x == 0 && blockIdx.x == 0) *dst = *src;
}

// W_k = (w - sum beta_q W_q) / ||.||, Z_k = z (the raw preconditioned
// vector) and the preconditioner's next input W_k, in precision P.  The
// residual is not touched per iteration: alpha_k = (W_k, r0) and the
// running norm are scalars (gcr_scalars), and r = r0 - sum alpha_q W_q is
// formed once per basis (k_gcr_rupdate), as is x (k_gcr_xupdate).  Per
// iteration this reads the basis W twice (the sums and here) and nothing of
// Z: about 2k + 7 vectors against 3k + 11 for the form that orthogonalised
// z and updated r every iteration.
//
// (16 bytes of each vector per thread; n is the padded length.  Memory bound:
// 1025 x 513 in FP32, 12 vectors on average, 12.1 us, 23.6 with 4-byte loads)
template <typename P>
__global__ void __launch_bounds__(256) k_gcr_finish(size_t n, int k, P *W, P *__restrict__ Z, const double *dots1,
                                                    const double *dots2, const double *sc, const P *z, const P *w,
                                                    P *__restrict__ pin) {
    typedef vec16<P> V;
    pdl_wait();
    __shared__ P bsh[GCR_MAX_M];
    const double *beta = sc[5] != 0.0 ? dots2 : dots1;
    for (int q = threadIdx.x; q < k; q += blockDim.x) bsh[q] = (P)beta[q];
    __syncthreads();
    const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * V::N;
    if (i >= n) return;
    // (a second pass left its vector in W_k)
    V ws = *reinterpret_cast<const V *>((sc[5] != 0.0 ? W + (size_t)k * n : w) + i);
    const V zi = *reinterpret_cast<const V *>(z + i);
#pragma unroll 4
    for (int q = 0; q < k; q++) {
        const V wq = *reinterpret_cast<const V *>(W + q * n + i);
#pragma unroll
        for (int e = 0; e < V::N; e++) ws.v[e] -= bsh[q] * wq.v[e];
    }
    const P s = (P)sc[0];
#pragma unroll
    for (int e = 0; e < V::N; e++) ws.v[e] *= s;
    *reinterpret_cast<V *>(W + (size_t)k * n + i) = ws;
    *reinterpret_cast<V *>(pin + i) = ws;
    *reinterpret_cast<V *>(Z + (size_t)k * n + i) = zi;
}

// r = r - sum alpha_q W_q over the basis (end of a basis); the P copy of the
// new r0 for the sums (rp, the FP32 form) and the preconditioner's input
template <typename P, typename T>
__global__ void k_gcr_rupdate(size_t n, int k, const P *__restrict__ W, const double *__restrict__ sc,
                              T *__restrict__ r, P *__restrict__ rp, P *__restrict__ pin) {
    __shared__ P ash[GCR_MAX_M];
    for (int q = threadIdx.x; q < k; q += blockDim.x) ash[q] = (P)sc[8 + q];
    __syncthreads();
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    P a = 0;
    for (int q = 0; q < k; q++) a += ash[q] * W[q * n + i];
    const T rn = (T)((double)r[i] - (double)a);
    r[i] = rn;
    if (rp) rp[i] = (P)rn;
    pin[i] = (P)rn;
}

// start of the solve: the P copy of r0 (FP32 form) and the first input
template <typename P, typename T>
__global__ void k_gcr_start(size_t n, const T *__restrict__ r, P *__restrict__ rp, P *__restrict__ pin) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const P v = (P)r[i];
    if (rp) rp[i] = v;
    pin[i] = v;
}

// x += sum_{q < k} gamma_q Z_q (gamma = U^-1 alpha, k_gcr_gamma): the basis
// part of the iterate, once per basis (at a restart and at the end)
template <typename P, typename T>
__global__ void k_gcr_xupdate(size_t n, int k, const P *__restrict__ Z, const double *__restrict__ gamma,
                              T *__restrict__ x) {
    __shared__ P ash[GCR_MAX_M];
    for (int q = threadIdx.x; q < k; q += blockDim.x) ash[q] = (P)gamma[q];
    __syncthreads();
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    P a = 0;
    for (int q = 0; q < k; q++) a += ash[q] * Z[q * n + i];
    x[i] = (T)((double)x[i] + (double)a);
}

template <typename T>
__global__ void k_axpby(size_t n, double a, const T *__restrict__ x, double b, T *__restrict__ y) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = (T)(a * (double)x[i] + b * (double)y[i]);
}

template <typename Tin, typename Tout>
__global__ void k_convert(size_t n, const Tin *__restrict__ a, Tout *__restrict__ b) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) b[i] = (Tout)a[i];
}

// Pressure gauge: the decoupled operator annihilates a constant pressure, but
// the rheology does not (pressure-dependent yield), so every correction is
// returned with zero mean over the pressure equations.

static mdz_status remove_pressure_mean(mdz_ctx *ctx, double *p, cudaStream_t st) {
    const mdz_dgrid &g = ctx->g;
    int np = g.ncx * g.ncz;
    double *d = (double *)(ctx->d_counters + 24);
    int blocks = mdz_blocks(np, 256);
    if (blocks > 152 * 4) blocks = 152 * 4;
    k_psum<double><<<blocks, 256, 0, st>>>(np, g.BCp, p, ctx->red_part + MDZ_RP_PSUM, ctx->red_cnt + MDZ_RC_PSUM, d);
    MDZ_LAUNCHED(ctx);
    k_psub<double><<<mdz_blocks(np), MDZ_THREADS, 0, st>>>(np, g.BCp, d, p);
    MDZ_LAUNCHED(ctx);
    return MDZ_OK;
}

// One Gram-Schmidt pass's sums in one launch: (w, W_q) for q < k, then
// (w, w) and (w, r) as vectors k and k + 1 (b = w), summed as k_dots does
// (the last block of each block row adds its row's partials in block order);
// the last row to finish (a second arrival counter) then runs the pass's
// scalar step: the check of the first pass (sc[5] = 1 asks for a second pass,
// else the scalars), or the scalars of the second.
// cnt[0]: rows finished, cnt[1 + y]: blocks of row y finished.
// SECOND: the second pass, whose vector is w - sum beta_q W_q with the first
// pass's sums beta; every block row forms it (all of W is read once per row, in
// the few iterations that need it), the first writes it to W_k, where the finish
// takes it from.  (As a launch of its own the correction cost every iteration a
// launch that returned at once, 1.5 us.)
template <typename T, int MDOT_Q, bool SECOND>
__global__ void __launch_bounds__(256) k_gcr_dots(int k, size_t n, const T *const *__restrict__ a,
                                                  const T *w, const T *r, T *W, const double *beta, double *part,
                                                  double *out, double *sc, double *tri, unsigned int *cnt,
                                                  double *note, double ticket) {
    typedef vec16<T> V;
    constexpr int mode = SECOND ? 2 : 1;
    pdl_wait();
    if (SECOND && sc[5] == 0.0) return;
    __shared__ double sh[dots_shared<T, MDOT_Q>()];
    const int nq = k + 2, q0 = blockIdx.y * MDOT_Q;
    const T *ap[MDOT_Q];
#pragma unroll
    for (int j = 0; j < MDOT_Q; j++) {
        const int q = q0 + j;
        ap[j] = q < k ? a[q] : (q == k ? w : (q == k + 1 ? r : nullptr));
    }
    double bs[MDOT_Q];
    if constexpr (SECOND) {
        __shared__ T bsh[GCR_MAX_M];
        for (int q = threadIdx.x; q < k; q += blockDim.x) bsh[q] = (T)beta[q];
        __syncthreads();
        const bool write = blockIdx.y == 0;
        dots_block<T, MDOT_Q>(nq, n, ap, [&](size_t i) {
            V ws = *reinterpret_cast<const V *>(w + i);
            for (int q = 0; q < k; q++) {
                const V wq = *reinterpret_cast<const V *>(W + q * n + i);
#pragma unroll
                for (int e = 0; e < V::N; e++) ws.v[e] -= bsh[q] * wq.v[e];
            }
            if (write) *reinterpret_cast<V *>(W + (size_t)k * n + i) = ws;
            return ws;
        }, k - q0, part, bs, sh);
    } else {
        dots_block<T, MDOT_Q>(nq, n, ap, [&](size_t i) { return *reinterpret_cast<const V *>(w + i); }, -1, part, bs, sh);
    }
    if (!mdz_arrive_last(cnt + 1 + blockIdx.y, gridDim.x)) return;
    const int nrow = nq - q0 < MDOT_Q ? nq - q0 : MDOT_Q;
    mdz_sum_partials(part + (size_t)q0 * gridDim.x, gridDim.x, nrow, out + q0);
    if (!mdz_arrive_last(cnt, gridDim.y)) return;
    if (threadIdx.x >= 32) return;
    // scalars of the iteration, one warp: lane q has d[q] and d[q + 32]
    static_assert(GCR_MAX_M <= 64, "two coefficients per lane");
    const int lane = threadIdx.x;
    const double d[2] = {lane < k ? __ldcg(out + lane) : 0.0, lane + 32 < k ? __ldcg(out + lane + 32) : 0.0};
    const double dk = __ldcg(out + k), dr = __ldcg(out + k + 1), dd = warp_sum_all(d[0] * d[0] + d[1] * d[1]);
    if (mode == 1) {
        // second pass when the first removed all but 1e-3 (FP64 basis) or 1e-1
        // (FP32 basis: its orthogonality decays faster, and alpha is taken
        // from r0 through the triangle) of w's squared norm
        if (k > 0 && !(dk - dd > (sizeof(T) == 4 ? 1e-1 : 1e-3) * dk)) {   // keep this pass's coefficients in U
            for (int h = 0; h < 2; h++)
                if (32 * h + lane < k) tri[(size_t)k * GCR_MAX_M + 32 * h + lane] = d[h];
            if (lane == 0) sc[5] = 1.0;
            return;
        }
        if (lane == 0) sc[5] = 0.0;
    }
    gcr_scalars(k, d, dk, dr, dd, sc, tri, mode == 2, note, ticket);
}

template <typename T>
static mdz_status gcr_dots_launch(mdz_ctx *ctx, gcr_space<T> &S, int k, const T *w, const T *r, const double *beta,
                                  double *out, double *sc, double ticket, cudaStream_t st) {
    if (beta)
        MDZ_PDL(ctx, (k_gcr_dots<T, dots_q<T>(), true>), dots_grid<T>(S.ld, k + 2), 256, 0, st, k, S.ld, S.dA0, w, r, S.W,
                beta, ctx->red_part + MDZ_RP_DOTS, out, sc, S.tri, ctx->red_cnt + MDZ_RC_GCR, ctx->solver->sc + GCR_NOTE,
                ticket);
    else
        MDZ_PDL(ctx, (k_gcr_dots<T, dots_q<T>(), false>), dots_grid<T>(S.ld, k + 2), 256, 0, st, k, S.ld, S.dA0, w, r, S.W,
                beta, ctx->red_part + MDZ_RP_DOTS, out, sc, S.tri, ctx->red_cnt + MDZ_RC_GCR, ctx->solver->sc + GCR_NOTE,
                ticket);
    return MDZ_OK;
}

template <typename T>
static mdz_status dots_launch(mdz_ctx *ctx, gcr_space<T> &S, int q0, int nq, const T *b, double *out,
                              cudaStream_t st) {
    if (nq <= 0) return MDZ_OK;
    k_dots<T, dots_q<T>()><<<dots_grid<T>(S.ld, nq), 256, 0, st>>>(nq, S.ld, S.dA0 + q0, b, ctx->red_part + MDZ_RP_DOTS,
                                                                   ctx->red_cnt + MDZ_RC_DOTS, out);
    MDZ_LAUNCHED(ctx);
    return MDZ_OK;
}

// The running norm of the iteration with this ticket, as gcr_scalars wrote it
// to host memory (GCR_NOTE), usually before the iteration's last launch ends.  The
// wait spins, as the runtime's own waits do by default; a process that asked for
// waits that block (cudaDeviceScheduleBlockingSync) or yield gets those.
static mdz_status gcr_wait_note(mdz_ctx *ctx, double ticket, cudaStream_t st, unsigned schedule, double *rn2) {
    volatile double *note = ctx->solver->sc + GCR_NOTE;
    if (schedule == cudaDeviceScheduleBlockingSync) MDZ_CUDA(ctx, cudaStreamSynchronize(st));
    for (long long spin = 1; note[1] != ticket; spin++) {
        if (schedule == cudaDeviceScheduleYield) std::this_thread::yield();
        if (spin % 4096) continue;
        const cudaError_t e = cudaStreamQuery(st);   // a failed launch never writes its ticket
        if (e == cudaErrorNotReady) continue;
        if (e != cudaSuccess) return mdz_cuda_check(ctx, e, "GCR iteration");
        if (note[1] != ticket) return mdz_fail(ctx, MDZ_ERR_STATE, "GCR: an iteration ended without its norm");
    }
    std::atomic_thread_fence(std::memory_order_acquire);
    *rn2 = note[0];
    return MDZ_OK;
}

// The preconditioner's ~10 launches per level, captured once per precision
// (its buffers, coefficients and the Krylov vectors r, z never move; the
// coefficients' values are refreshed by mg_setup outside the graph).
template <typename T>
static mdz_status precond_graph(mdz_ctx *ctx, gcr_space<T> &S, mg_hier<T> &H, const double *eta_n, const T *Dt,
                                cudaStream_t st, cudaGraphExec_t *out, long long *launches, int *slot_out) {
    mdz_solver *SV = ctx->solver;
    const int slot = (sizeof(T) == 8 ? 0 : 2) + (H.newton ? 1 : 0) + (Dt ? 4 : 0);
    *slot_out = slot;
    if (SV->pre[slot] && SV->pre_eta[slot] == eta_n) {
        *out = SV->pre[slot];
        *launches = SV->pre_launches[slot];
        return MDZ_OK;
    }
    if (SV->pre[slot]) { cudaGraphExecDestroy(SV->pre[slot]); SV->pre[slot] = nullptr; }
    const long long l0 = ctx->launches;
    MDZ_CUDA(ctx, cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    mdz_status s = precondition<T>(ctx, H, Dt, S.pin, S.z, S.nu, S.nv, st);
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamEndCapture(st, &g);
    if (s != MDZ_OK) { if (g) cudaGraphDestroy(g); return s; }
    if (e != cudaSuccess) return mdz_cuda_check(ctx, e, "preconditioner capture");
    e = cudaGraphInstantiate(&SV->pre[slot], g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) { SV->pre[slot] = nullptr; return mdz_cuda_check(ctx, e, "preconditioner graph"); }
    SV->pre_launches[slot] = ctx->launches - l0;
    SV->pre_eta[slot] = eta_n;
    {   // per level: nu1 + nu2 sweeps and one residual, each reading x, f, the
        // inverse diagonal and both viscosities and writing one vector, plus
        // the tags; restriction and prolongation one read + one write each;
        // the fine-level pressure block and right-hand side 3 vectors
        double b = 0.0;
        for (int l = 0; l < H.nlev; l++) {
            const mg_level<T> &L = H.L[l];
            double nuv = (double)(L.nu() + L.nv()), nc = (double)L.ncx * L.ncz, ng = (double)L.Nx * L.Nz;
            b += (SV->nu1 + SV->nu2 + 1) * (sizeof(T) * (4.0 * nuv + nc + ng) + (nuv + nc + ng));
            b += 4.0 * sizeof(T) * nuv;
        }
        b += 3.0 * sizeof(T) * (double)S.n;
        if (Dt) b += sizeof(T) * (double)S.np;
        SV->pre_bytes[slot] = b;
    }
    ctx->launches = l0;
    *out = SV->pre[slot];
    *launches = SV->pre_launches[slot];
    return MDZ_OK;
}

// ---------------------------------------------------------------------------
// GCR on K x = b (x0 = 0), right-preconditioned.  The preconditioner
// (V-cycle), the operator apply and the stored basis Z, W run in precision
// P; the iterate x, the residual r and every inner product are FP64 (T).
// P = T = double: the plain FP64 solve.  T = double, P = float: the inner
// solve of the FP32 form (r narrowed to FP32 before the preconditioner), whose
// recursive residual differs from b - K x only by FP32 rounding of the
// applies and basis vectors, which the FP64 defect correction outside absorbs.
template <typename T, typename P>
static mdz_status gcr_solve(mdz_ctx *ctx, gcr_space<T> &S, gcr_space<P> &SP, mg_hier<P> &H,
                            const stokes_coefs<P> &K, bool newton, const double *eta_n, double rtol, int maxit,
                            int *its_out, double *rel_out, cudaStream_t st) {
    constexpr bool mixed = sizeof(T) != sizeof(P);
    mdz_solver *SV = ctx->solver;
    stokes_geom G = mdz_stokes_geom(ctx);
    // vector kernels run over the padded length (zeros beyond the n unknowns)
    const size_t n = S.ld, nu = S.nu, nv = S.nv;
    int nb = mdz_blocks(n);
    const int nb16 = mdz_blocks((long long)n, 256 * vec16<P>::N);
    MDZ_CUDA(ctx, cudaMemsetAsync(S.x, 0, sizeof(T) * n, st));
    // ||r0||
    // S.dots layout (doubles, B = GCR_MAX_M + 8): first-pass sums at 0, the
    // scalars sc at GCR_MAX_M + 4, second-pass sums at 2B, a scratch sum at 3B
    const int B = GCR_MAX_M + 8;
    double *const d1 = S.dots, *const sc = d1 + (GCR_MAX_M + 4), *const d2 = d1 + 2 * B, *const dots = d1 + 3 * B;
    MDZ_CUDA(ctx, cudaMemsetAsync(S.dots, 0, sizeof(double) * 4 * B, st));
    mdz_status s;
    cudaGraphExec_t pre = nullptr;
    long long pre_launches = 0;
    int pslot = 0;
    const P *Dt = newton && SV->schur == 1 ? K.D11 : nullptr;   // tangent Schur scaling (Newton solves)
    if ((s = precond_graph<P>(ctx, SP, H, eta_n, Dt, st, &pre, &pre_launches, &pslot)) != MDZ_OK) return s;
    // (r, r) via the pointer-table slot m+1 against r itself
    if ((s = dots_launch<T>(ctx, S, S.m + 1, 1, S.r, dots, st)) != MDZ_OK) return s;
    k_set_scalar<<<1, 32, 0, st>>>(sc + 3, dots);
    MDZ_LAUNCHED(ctx);
    MDZ_CUDA(ctx, cudaMemcpyAsync(SV->sc, dots, sizeof(double), cudaMemcpyDeviceToHost, st));
    MDZ_CUDA(ctx, cudaStreamSynchronize(st));
    {
        const volatile int *flags = (const volatile int *)(SV->sc + 20);
        if (flags[0]) return mdz_fail(ctx, MDZ_ERR_NOT_CONVERGED, "multigrid: coarsest-level block singular");
        if (flags[1]) return mdz_fail(ctx, MDZ_ERR_STATE, "multigrid: Galerkin entry outside the stencil footprint");
    }
    double rn2 = SV->sc[0], rn02 = rn2;
    int it = 0;
    if (rn02 == 0.0) { if (its_out) *its_out = 0; if (rel_out) *rel_out = 0.0; return MDZ_OK; }
    // the preconditioner's first input r0 and (FP32 form) the FP32 copy of r0
    k_gcr_start<P, T><<<nb, MDZ_THREADS, 0, st>>>(n, S.r, mixed ? SP.r : (P *)nullptr, SP.pin);
    MDZ_LAUNCHED(ctx);
    int k = 0;
    const double *gamma = SP.tri + (size_t)GCR_MAX_M * GCR_MAX_M;
    // end of a basis: x += Z U^-1 alpha, r = r0 - W alpha (and its copies)
    auto end_basis = [&](bool need_r) -> mdz_status {
        if (k == 0) return MDZ_OK;
        k_gcr_gamma<<<1, 32, 0, st>>>(k, sc, SP.tri);
        MDZ_LAUNCHED(ctx);
        k_gcr_xupdate<P, T><<<nb, MDZ_THREADS, 0, st>>>(n, k, SP.Z, gamma, S.x);
        MDZ_LAUNCHED(ctx);
        if (need_r) {
            k_gcr_rupdate<P, T><<<nb, MDZ_THREADS, 0, st>>>(n, k, SP.W, sc, S.r, mixed ? SP.r : (P *)nullptr, SP.pin);
            MDZ_LAUNCHED(ctx);
        }
        k = 0;
        return MDZ_OK;
    };
    const int check = SV->check > 0 ? SV->check : 1;
    unsigned schedule = 0;
    MDZ_CUDA(ctx, cudaGetDeviceFlags(&schedule));
    for (it = 0; it < maxit; it++) {
        if (k == S.m && (s = end_basis(true)) != MDZ_OK) return s;   // restart: fold the basis into x and r
        cudaEvent_t ev;
        mdz_prof_begin(ctx, MDZ_PROF_MG_SMOOTH, st, &ev);
        MDZ_CUDA(ctx, cudaGraphLaunch(pre, st));
        ctx->launches += pre_launches;
        mdz_prof_end(ctx, MDZ_PROF_MG_SMOOTH, SV->pre_bytes[pslot], st, ev);
        mdz_prof_begin(ctx, MDZ_PROF_STOKES_APPLY, st, &ev);
        stokes_apply_launch<P>(G, K, stokes_cvec<P>{SP.z, SP.z + nu, SP.z + nu + nv},
                               stokes_vec<P>{SP.w, SP.w + nu, SP.w + nu + nv}, nullptr, newton, true, st);
        MDZ_LAUNCHED(ctx);
        {   // algorithmic bytes: input and output vectors, the D-tensor read once, tags
            size_t nc = S.np, ng = (size_t)G.Nx * G.Nz;
            double coef = newton ? (8.0 * nc + 4.0 * ng) : (2.0 * nc + ng);
            double bytes = sizeof(P) * (2.0 * S.n + coef) + (double)(nu + nv + nc + ng);
            mdz_prof_end(ctx, MDZ_PROF_STOKES_APPLY, bytes, st, ev);
        }
        mdz_prof_begin(ctx, MDZ_PROF_KRYLOV, st, &ev);
        // The basis W and the raw preconditioned vectors Z stay in the apply's
        // precision P (in the FP32 form: as the FP32 V-cycle and apply
        // produced them); x, r and every sum are FP64.  First pass:
        // (w, W_q) q < k, (w, w), (w, r0); the check decides on the device
        // whether a second pass runs.
        SV->ticket += 1.0;
        if ((s = gcr_dots_launch<P>(ctx, SP, k, SP.w, SP.r, nullptr, d1, sc, SV->ticket, st)) != MDZ_OK) return s;
        // second pass (returns at once unless sc[5] = 1)
        if (k > 0 && (s = gcr_dots_launch<P>(ctx, SP, k, SP.w, SP.r, d1, d2, sc, SV->ticket, st)) != MDZ_OK) return s;
        MDZ_PDL(ctx, k_gcr_finish<P>, nb16, 256, 0, st, n, k, SP.W, SP.Z, d1, d2, sc, SP.z, SP.w, SP.pin);
        {   // algorithmic bytes (one Gram-Schmidt pass): the sums read W_q,
            // w and r0 (k + 2 P vectors); the finish reads W_q, w, z and
            // writes W_k, Z_k and the next input (k + 5)
            double pv = 2.0 * k + 7.0;
            mdz_prof_end(ctx, MDZ_PROF_KRYLOV, (double)S.n * sizeof(P) * pv, st, ev);
        }
        k++;
        // the running norm lives on the device; the host looks every `check`
        // iterations, at each restart and at the iteration limit
        if ((it + 1) % check != 0 && k != S.m && it + 1 < maxit) continue;
        if ((s = gcr_wait_note(ctx, SV->ticket, st, schedule & cudaDeviceScheduleMask, &rn2)) != MDZ_OK) return s;
        if (!std::isfinite(rn2)) return mdz_fail(ctx, MDZ_ERR_NAN, "GCR: NaN in the Krylov iteration");
        if (rn2 <= rtol * rtol * rn02 || (k == S.m)) {
            // fold the basis in and take the true norm of r at convergence
            // and at each restart
            if ((s = end_basis(true)) != MDZ_OK) return s;
            if ((s = dots_launch<T>(ctx, S, S.m + 1, 1, S.r, dots, st)) != MDZ_OK) return s;
            k_set_scalar<<<1, 32, 0, st>>>(sc + 3, dots);
            MDZ_LAUNCHED(ctx);
            MDZ_CUDA(ctx, cudaMemcpyAsync(SV->sc, dots, sizeof(double), cudaMemcpyDeviceToHost, st));
            MDZ_CUDA(ctx, cudaStreamSynchronize(st));
            rn2 = SV->sc[0];
            if (rn2 <= rtol * rtol * rn02) { it++; break; }
        }
    }
    if ((s = end_basis(false)) != MDZ_OK) return s;   // the current basis' part of the iterate
    if (its_out) *its_out = it;
    if (rel_out) *rel_out = sqrt(rn2 > 0 ? rn2 : 0.0) / sqrt(rn02);
    return MDZ_OK;
}

// ---------------------------------------------------------------------------
// Public device-level solve: K dx = F.  F and dx in grid layout (u | v | p
// contiguous, length n), FP64.  precision 64: plain FP64 GCR + FP64 V-cycle;
// precision 32: FP64 defect correction around FP32 GCR + FP32 V-cycle.
mdz_status mdz_dev_solve(mdz_ctx *ctx, const mdz_fields &f, bool newton, int precision, double rtol, int maxit,
                         const double *F, double *dx, mdz_solve_stats *stats, cudaStream_t st, bool reuse_mg) {
    mdz_status s = mdz_solver_ensure(ctx);
    if (s != MDZ_OK) return s;
    mdz_solver *SV = ctx->solver;
    gcr_space<double> &S64 = SV->g64;
    const size_t n = S64.n, nu = S64.nu, nv = S64.nv;
    stokes_geom G = mdz_stokes_geom(ctx);
    stokes_coefs<double> K64 = mdz_coefs64(f);
    int its = 0, total = 0, cycles = 0;
    double rel = 1.0;
    if (precision == 64) {
        const bool nh = newton && SV->mg_jacobian;
        if (!(reuse_mg && SV->mg64.built && SV->mg64.newton == nh))
            if ((s = mg_setup<double>(ctx, SV->mg64, f.eta_n, f.eta_s, K64, nh, st)) != MDZ_OK) return s;
        MDZ_CUDA(ctx, cudaMemcpyAsync(S64.r, F, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
        if ((s = gcr_solve<double, double>(ctx, S64, S64, SV->mg64, K64, newton, f.eta_n, rtol, maxit, &its, &rel,
                                           st)) != MDZ_OK)
            return s;
        MDZ_CUDA(ctx, cudaMemcpyAsync(dx, S64.x, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
        total = its;
        cycles = 1;
    } else {
        gcr_space<float> &S32 = SV->g32;
        // FP32 copy of the operator
        const double *Dsrc[12] = {f.D11_n, f.D12_n, f.D13_n, f.D14_n, f.D21_n, f.D22_n, f.D23_n, f.D24_n,
                                  f.D31_s, f.D32_s, f.D33_s, f.D34_s};
        for (int q = 0; q < 12; q++) {
            size_t m = q < 8 ? S32.np : (size_t)ctx->g.Nx * ctx->g.Nz;
            if (!newton && q != 0 && q != 5 && q != 10) continue;
            k_convert<double, float><<<mdz_blocks(m), MDZ_THREADS, 0, st>>>(m, Dsrc[q], S32.Dc[q]);
            MDZ_LAUNCHED(ctx);
        }
        stokes_coefs<float> K32{S32.Dc[0], S32.Dc[1], S32.Dc[2], S32.Dc[3], S32.Dc[4], S32.Dc[5], S32.Dc[6],
                                S32.Dc[7], S32.Dc[8], S32.Dc[9], S32.Dc[10], S32.Dc[11]};
        const bool nh = newton && SV->mg_jacobian;
        if (!(reuse_mg && SV->mg32.built && SV->mg32.newton == nh))
            if ((s = mg_setup<float>(ctx, SV->mg32, f.eta_n, f.eta_s, K32, nh, st)) != MDZ_OK) return s;
        // defect correction: r64 = F - K64 dx64 ; solve K32 e = r64 ; dx64 += e
        MDZ_CUDA(ctx, cudaMemsetAsync(dx, 0, sizeof(double) * n, st));
        MDZ_CUDA(ctx, cudaMemcpyAsync(S64.r, F, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
        double *dn = (double *)(ctx->d_counters + 8);
        double r0 = -1.0, prev = 1e300;
        auto defect = [&]() -> mdz_status {   // r64 = F - K64 dx
            stokes_apply_launch<double>(G, K64, stokes_cvec<double>{dx, dx + nu, dx + nu + nv},
                                        stokes_vec<double>{S64.t, S64.t + nu, S64.t + nu + nv}, nullptr, newton, true, st);
            MDZ_LAUNCHED(ctx);
            MDZ_CUDA(ctx, cudaMemcpyAsync(S64.r, F, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
            k_axpby<double><<<mdz_blocks(n), MDZ_THREADS, 0, st>>>(n, -1.0, S64.t, 1.0, S64.r);
            MDZ_LAUNCHED(ctx);
            return MDZ_OK;
        };
        // Each cycle solves for the current FP64 defect in FP32.  An FP32 solve
        // cannot resolve corrections whose K-image is below FP32 rounding of the
        // stresses, so the contraction per cycle degrades on stiff problems: the
        // loop runs while the defect still shrinks by 10 % and takes back a
        // cycle that made it grow.
        for (cycles = 0; cycles < 60; cycles++) {
            // norm of the FP64 defect
            if ((s = dots_launch<double>(ctx, S64, S64.m + 1, 1, S64.r, dn, st)) != MDZ_OK) return s;
            MDZ_CUDA(ctx, cudaMemcpyAsync(SV->sc + 8, dn, sizeof(double), cudaMemcpyDeviceToHost, st));
            MDZ_CUDA(ctx, cudaStreamSynchronize(st));
            double rn = sqrt(SV->sc[8]);
            if (r0 < 0) r0 = rn;
            rel = r0 > 0 ? rn / r0 : 0.0;
            if (rel <= rtol || r0 == 0.0) break;
            if (cycles > 0 && rel > prev) {   // the last correction made it worse: undo it
                k_axpby<double><<<mdz_blocks(n), MDZ_THREADS, 0, st>>>(n, -1.0, S64.x, 1.0, dx);
                MDZ_LAUNCHED(ctx);
                if ((s = defect()) != MDZ_OK) return s;
                rel = prev;
                break;
            }
            if (rel > 0.9 * prev || total >= maxit) break;   // refinement stalled or budget spent
            prev = rel;
            // Inner solve on the FP64 defect: FP64 Krylov space, FP32 stencils
            // and V-cycles.  The recursive residual differs from b - K64 x by
            // the FP32 rounding of the applies times the cancellation in the
            // Krylov sums, so each inner solve asks for at most three digits
            // and one basis length; the FP64 cycles carry the accuracy.
            double inner_rtol = rtol / rel;
            if (inner_rtol < 1e-3) inner_rtol = 1e-3;
            if (inner_rtol > 0.1) inner_rtol = 0.1;
            const int inner_max = maxit - total < S64.m ? maxit - total : S64.m;
            if ((s = gcr_solve<double, float>(ctx, S64, S32, SV->mg32, K32, newton, f.eta_n, inner_rtol, inner_max,
                                              &its, nullptr, st)) != MDZ_OK)
                return s;
            total += its;
            k_axpby<double><<<mdz_blocks(n), MDZ_THREADS, 0, st>>>(n, 1.0, S64.x, 1.0, dx);
            MDZ_LAUNCHED(ctx);
            if ((s = defect()) != MDZ_OK) return s;
        }
    }
    if ((s = remove_pressure_mean(ctx, dx + nu + nv, st)) != MDZ_OK) return s;
    if (stats) {
        stats->iterations = total;
        stats->refinements = cycles;
        stats->rel_residual = rel;
        stats->mg_levels = SV->mg64.nlev;
    }
    return MDZ_OK;
}

// ---------------------------------------------------------------------------
extern "C" mdz_status mdz_SolveStokesDefect(mdz_ctx *ctx, mdz_fields *f, int jacobian, int precision, double rtol,
                                            int maxit, const double *Fu, const double *Fv, const double *Fp,
                                            double *dxu, double *dxv, double *dxp, int *iterations,
                                            double *rel_residual) {
    if (!ctx || !f || !Fu || !Fv || !Fp || !dxu || !dxv || !dxp)
        return ctx ? mdz_fail(ctx, MDZ_ERR_ARG, "SolveStokesDefect: null argument") : MDZ_ERR_ARG;
    if (precision != 64 && precision != 32) return mdz_fail(ctx, MDZ_ERR_ARG, "SolveStokesDefect: precision 64 or 32");
    mdz_status s = mdz_ensure_fields(ctx);
    if (s != MDZ_OK) return s;
    if ((s = mdz_solver_ensure(ctx)) != MDZ_OK) return s;
    cudaStream_t st = ctx->stream;
    if ((s = mdz_upload_fields(ctx, f, st)) != MDZ_OK) return s;
    const mdz_dgrid &g = ctx->g;
    size_t nu = (size_t)g.Nx * (g.Nz + 1), nv = (size_t)(g.Nx + 1) * g.Nz, np = (size_t)g.ncx * g.ncz;
    double *buf = (double *)mdz_stage(ctx, 7, sizeof(double) * 2 * (nu + nv + np));
    if (!buf) return mdz_fail(ctx, MDZ_ERR_CUDA, "SolveStokesDefect: staging allocation failed");
    double *F = buf, *dx = buf + nu + nv + np;
    MDZ_CUDA(ctx, cudaMemcpyAsync(F, Fu, nu * 8, cudaMemcpyHostToDevice, st));
    MDZ_CUDA(ctx, cudaMemcpyAsync(F + nu, Fv, nv * 8, cudaMemcpyHostToDevice, st));
    MDZ_CUDA(ctx, cudaMemcpyAsync(F + nu + nv, Fp, np * 8, cudaMemcpyHostToDevice, st));
    mdz_solve_stats stt{};
    if ((s = mdz_dev_solve(ctx, ctx->d, jacobian != 0, precision, rtol, maxit, F, dx, &stt, st)) != MDZ_OK) return s;
    MDZ_CUDA(ctx, cudaMemcpyAsync(dxu, dx, nu * 8, cudaMemcpyDeviceToHost, st));
    MDZ_CUDA(ctx, cudaMemcpyAsync(dxv, dx + nu, nv * 8, cudaMemcpyDeviceToHost, st));
    MDZ_CUDA(ctx, cudaMemcpyAsync(dxp, dx + nu + nv, np * 8, cudaMemcpyDeviceToHost, st));
    MDZ_CUDA(ctx, cudaStreamSynchronize(st));
    if (iterations) *iterations = stt.iterations;
    if (rel_residual) *rel_residual = stt.rel_residual;
    if (!(stt.rel_residual <= rtol))
        return mdz_fail(ctx, MDZ_ERR_NOT_CONVERGED, "SolveStokesDefect: relative residual %.3e > %.3e after %d its",
                        stt.rel_residual, rtol, stt.iterations);
    return MDZ_OK;
}
