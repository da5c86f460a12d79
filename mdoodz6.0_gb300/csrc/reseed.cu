// Marker reseeding: the reseeding half of CountPartCell (RESEED = 1,
// SOURCE/ParticleRoutines.c:3543-4480) on the resident markers, with the
// result the reference gives on one OpenMP thread.
//
//   quarter cells  the grid extended by one cell on each side, split into
//                  (2 (Ncx + 2)) x (2 (Ncz + 2)) quarter cells; an active
//                  marker's quarter cell is ceil(((x - (xc_e0 - dx/4)) / dx) 2
//                  + 0.5) - 1, clamped (:3905-3921), counted and listed in
//                  ascending marker index (a stable counting sort: count,
//                  scan, scatter, per-bin index sort);
//   deficiency     each quarter cell of the inner region whose centroid is not
//                  air and that holds fewer than (int)(ceil(min_part_cell) / 4)
//                  markers gets one marker at its centre (AddPartCell2
//                  :977-1030); every such cell is independent of the others,
//                  one thread each;
//   neighbour      the new marker copies the nearest marker of the 5x5 quarter
//                  cells around it, visited in the reference's order
//                  (:4105-4283) and replaced only by a strictly closer one
//                  (FindClosestPhase2 :841-890);
//   slots          new markers are numbered quarter-column by quarter-column
//                  (the reference's k-outer, l-inner loop); the first ones
//                  take the slots of inactive markers in index order, the
//                  rest are appended (:4285-4330): two scans;
//   properties     phase, velocity and strains are copied, T, P and the stresses
//                  copied (DirectNeighbour = 1) or interpolated from the grid
//                  (Centers2Particle :259-455, Vertices2Particle :461-520)
//                  (AssignMarkerProperties :648-762).  The cohesion multiplier
//                  travels with the copied marker.
//
// Sources of a copy are active markers, destinations inactive slots or slots
// past the old count: no thread reads what another writes.  Index arithmetic
// rounds every product before its sum (__dmul_rn / __dadd_rn) so that no
// contraction moves a marker to another quarter cell.  Distances square with
// a * a where the reference calls pow(a, 2); the two can differ in the last
// bit, so a nearest-marker choice can differ only between two candidates whose
// distances agree to one unit in the last place.
#include <cmath>
#include "mdz_internal.cuh"

struct mdz_reseed_ws {
    long long cap = 0;
    int nq = 0, ni = 0;
    int *qcell = nullptr, *qsorted = nullptr;            // per marker
    int *qcount = nullptr, *qstart = nullptr, *qpart = nullptr;   // per quarter cell
    int *flag = nullptr, *rank = nullptr, *src = nullptr, *ipart = nullptr;           // per inner quarter cell
    int *inact = nullptr, *islot = nullptr, *reuse = nullptr, *mpart = nullptr;       // per marker
    int *status = nullptr;                               // [0] no-neighbour flag, [1] a marker without a position code
};

void mdz_reseed_free(mdz_ctx *ctx) {
    mdz_reseed_ws *W = ctx->reseed;
    if (!W) return;
    int *p[] = {W->qcell, W->qsorted, W->qcount, W->qstart, W->qpart, W->flag, W->rank,
                W->src, W->ipart, W->inact, W->islot, W->reuse, W->mpart, W->status};
    for (int *q : p)
        if (q) cudaFree(q);
    delete W;
    ctx->reseed = nullptr;
}

// Position code of a marker for the window search: its two coordinates in
// quarter cells, 13 fractional bits, modulo 8 (16 bits each).  The difference of
// two codes in one window (5 x 5 quarter cells) is their distance in 16-bit
// arithmetic.
constexpr double RS_UNIT = 8192.0;

// Quarter-grid geometry, every constant formed as the reference forms it.
struct quarter_geom {
    int nxl, nzl, Ncx, Ncz, Nx;
    double dx, dz, idx2, idz2, xge, zge, qx0, qz0;   // extended vertex origin; quarter-index origin xc_e0 - dx/4
    double xg0, zg0, xmin, xmax, zmin, zmax;
    float cx, cz, width;   // window search: squares of dx, dz over the larger; box width in its units
};

static quarter_geom make_quarter_geom(const mdz_ctx *ctx) {
    const mdz_grid_desc &d = ctx->host_desc;
    quarter_geom q;
    q.Ncx = d.Nx - 1; q.Ncz = d.Nz - 1; q.Nx = d.Nx;
    q.nxl = 2 * (q.Ncx + 2); q.nzl = 2 * (q.Ncz + 2);
    q.dx = d.dx; q.dz = d.dz;
    q.idx2 = 2.0 / d.dx; q.idz2 = 2.0 / d.dz;
    q.xg0 = d.xg[0]; q.zg0 = d.zg[0];
    q.xge = q.xg0 - q.dx;
    q.zge = q.zg0 - q.dz;
    const double xce = 0.5 * (q.xge + (q.xge + q.dx)), zce = 0.5 * (q.zge + (q.zge + q.dz));
    q.qx0 = xce - q.dx / 4.0;
    q.qz0 = zce - q.dz / 4.0;
    q.xmin = d.xmin; q.xmax = d.xmax; q.zmin = d.zmin; q.zmax = d.zmax;
    const double big = q.dx > q.dz ? q.dx : q.dz;
    q.cx = (float)((q.dx / big) * (q.dx / big));
    q.cz = (float)((q.dz / big) * (q.dz / big));
    q.width = (float)((q.xmax - q.xmin) / (0.5 * big) * RS_UNIT);
    return q;
}

// ceil(v + 0.5) - 1 of the reference's nearest-node formula, as an int
__device__ __forceinline__ int nearest_of(double v) { return (int)(ceil(__dadd_rn(v, 0.5)) - 1.0); }

// Quarter-cell index of a marker at distance d from the first quarter line, by
// the mantissa where the roundings cannot matter (2^-19 of a quarter cell from a
// line), by the reference's quotient, product and sum elsewhere; the position
// code's 16 bits from the same mantissa.  False: outside the quarter grid, or
// not a number (no code).
__device__ __forceinline__ bool quarter_index(double d, double h, double ih2, int n, int &i, unsigned &code) {
    const unsigned long long t = (unsigned long long)__double_as_longlong(__fma_rn(d, ih2, 0.5 + 6442450944.0));
    if (!line_index(d, ih2, 0.5, i)) i = nearest_of(__dmul_rn(__ddiv_rn(d, h), 2.0));
    code = (unsigned)(t >> 7) & 0xffffu;
    const bool in = i >= 0 && i < n && (unsigned)(t >> 52) == 0x41Fu;
    i = i < 0 ? 0 : (i > n - 1 ? n - 1 : i);
    return in;
}

__global__ void k_quarter_count(int n, const double *__restrict__ x, const double *__restrict__ z,
                                const int *__restrict__ phase, quarter_geom q, int *__restrict__ qcell,
                                int *__restrict__ code, int *__restrict__ arrival, int *__restrict__ qcount,
                                int *__restrict__ status) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    if (phase[k] < 0) { qcell[k] = -1; return; }
    int ic, jc;
    unsigned cx, cz;
    const bool in = quarter_index(x[k] - q.qx0, q.dx, q.idx2, q.nxl, ic, cx);
    if (!(quarter_index(z[k] - q.qz0, q.dz, q.idz2, q.nzl, jc, cz) && in)) status[1] = 1;   // exact searches only
    const int c = ic + jc * q.nxl;
    qcell[k] = c;
    code[k] = (int)(cx | cz << 16);
    arrival[k] = atomicAdd(&qcount[c], 1);
}

// Ascending marker index inside each quarter cell, and the codes in that order.
__global__ void k_quarter_sort(int nq, const int *__restrict__ start, int *__restrict__ sorted,
                               const int *__restrict__ code, int *__restrict__ qcode) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nq) return;
    const int b = start[c], e = start[c + 1];
    for (int i = b + 1; i < e; i++) {
        const int v = sorted[i];
        int j = i - 1;
        while (j >= b && sorted[j] > v) { sorted[j + 1] = sorted[j]; j--; }
        sorted[j + 1] = v;
    }
    for (int i = b; i < e; i++) qcode[i] = code[sorted[i]];
}

// New-marker position of inner quarter cell (k, l): xg[0] + ic dx/2 + dx/4 with
// ic = k - 2 (halving and quartering are exact as products with 0.5, 0.25).
__device__ __forceinline__ double new_pos(double o, int i, double h) {
    return __dadd_rn(__dadd_rn(o, __dmul_rn(__dmul_rn((double)i, h), 0.5)), __dmul_rn(h, 0.25));
}

// One thread per inner quarter cell; t runs over (k, l) with k fastest, the
// flags are stored in the reference's creation order q = (k-2) (nzl-4) + (l-2).
// The count test comes first (integer), then the air test of the cell's
// centroid, the neighbour count and the box test of the new position.
__global__ void k_reseed_cells(quarter_geom q, const signed char *__restrict__ tagp, const int *__restrict__ qstart,
                               int thr, int *__restrict__ flag, int *__restrict__ status) {
    const int wi = q.nxl - 4, wj = q.nzl - 4;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= wi * wj) return;
    const int k = 2 + t % wi, l = 2 + t / wi, qo = (k - 2) * wj + (l - 2), kd = k + l * q.nxl;
    int f = 0;
    if (qstart[kd + 1] - qstart[kd] < thr) {
        // centroid nearest to the quarter cell's centre, for the air test: the centre lies a quarter of a
        // cell from it, so nearest_of((centre - xc0) / dx) is k / 2 - 1 whatever the roundings
        int ic = (k >> 1) - 1, jc = (l >> 1) - 1;
        ic = ic < 0 ? 0 : (ic > q.Ncx - 1 ? q.Ncx - 1 : ic);
        jc = jc < 0 ? 0 : (jc > q.Ncz - 1 ? q.Ncz - 1 : jc);
        if (tagp[ic + jc * q.Ncx] != 30) {
            int neighs = 0;
#pragma unroll
            for (int w = -2; w <= 2; w++)   // the five cells of a row are one run
                neighs += qstart[kd + w * q.nxl + 3] - qstart[kd + w * q.nxl - 2];
            if (neighs == 0) {
                atomicOr(status, 1);
            } else {
                const double xn = new_pos(q.xg0, k - 2, q.dx), zn = new_pos(q.zg0, l - 2, q.dz);
                f = xn > q.xmin && zn > q.zmin && zn < q.zmax;
            }
        }
    }
    flag[qo] = f;
}

// Inverse of the ranks: list[rank] = quarter cell, so that the search below
// runs one thread per new marker.
__global__ void k_reseed_list(int ni, const int *__restrict__ flag, const int *__restrict__ rank,
                              int *__restrict__ list) {
    const int qo = blockIdx.x * blockDim.x + threadIdx.x;
    if (qo < ni && flag[qo]) list[rank[qo]] = qo;
}

__global__ void k_inactive_flags(int n, const int *__restrict__ phase, int *__restrict__ inact) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) inact[k] = phase[k] == -1 ? 1 : 0;
}

__global__ void k_inactive_list(int n, const int *__restrict__ inact, const int *__restrict__ islot,
                                int *__restrict__ reuse) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n && inact[k]) reuse[islot[k]] = k;
}

// Centers2Particle, non-periodic (SOURCE/ParticleRoutines.c:259-455): bilinear
// on the ghosted centroid lines, a column or row outside the centroids repeating
// the edge's (the reference's edge and corner folds); or, with vert,
// Vertices2Particle (:461-520): bilinear on the vertices.  One body for both, so
// that the lanes of a group take one field each in the same instructions.
__device__ __forceinline__ double grid_to_new(const mdz_dgrid &g, double x, double z, bool vert,
                                              const double *__restrict__ F) {
    const double dx = g.dx, dz = g.dz;
    const double *X = vert ? g.xg : g.xvz, *Z = vert ? g.zg : g.zvx;
    double dX = x - X[0], dZ = z - Z[0];
    if (vert) { dX = fabs(dX); dZ = fabs(dZ); }
    int j, i;
    if (!line_index(dX, g.idx, 0.0, j)) j = (int)(ceil(dX / dx) - 1.0);
    if (!line_index(dZ, g.idz, 0.0, i)) i = (int)(ceil(dZ / dz) - 1.0);
    const int nx = vert ? g.Nx : g.ncx, nz = vert ? g.Nz : g.ncz;
    int jw = j, je = j + 1, is = i, in_ = i + 1;
    if (!vert) {
        if (j < 0 || j > nx || i < 0 || i > nz) return 0.0;   // outside the ghosted frame: new markers lie inside the box
        jw = j > 0 ? j - 1 : 0; je = j < nx ? j : nx - 1;
        is = i > 0 ? i - 1 : 0; in_ = i < nz ? i : nz - 1;
    }
    const int iSW = jw + is * nx, iSE = je + is * nx, iNW = jw + in_ * nx, iNE = je + in_ * nx;
    const double ax = (x - X[j]) / dx, az = (z - Z[i]) / dz;
    const signed char *t = vert ? g.BCg : g.BCp;
    auto rock = [](signed char v) { return v != 30 && v != 31; };
    if (rock(t[iSW]) && rock(t[iSE]) && rock(t[iNW]) && rock(t[iNE])) {   // the weights sum to 1: no quotient
        const double bx = 1.0 - ax, bz = 1.0 - az;
        return bz * (bx * F[iSW] + ax * F[iSE]) + az * (bx * F[iNW] + ax * F[iNE]);
    }
    double val = 0.0, sw = 0.0, w;
    if (t[iSW] != 30 && t[iSW] != 31) { w = (1.0 - ax) * (1.0 - az); val += w * F[iSW]; sw += w; }
    if (t[iSE] != 30 && t[iSE] != 31) { w = ax * (1.0 - az); val += w * F[iSE]; sw += w; }
    if (t[iNW] != 30 && t[iNW] != 31) { w = (1.0 - ax) * az; val += w * F[iNW]; sw += w; }
    if (t[iNE] != 30 && t[iNE] != 31) { w = ax * az; val += w * F[iNE]; sw += w; }
    return sw > 1e-13 ? val / sw : val;
}

struct reseed_fields {
    const double *T_n, *sxxd_n, *szzd_n, *sxz_s, *p_n;
};

// Place of window cell (dk, dl), at [(dl + 2) 5 + dk + 2], in the order in which
// AddPartCell2's neighbour list visits them: the cell, its four neighbours (W, E,
// S, N) and corners (SW, SE, NW, NE), the same at two cells' distance, and the
// remaining eight by rows (dl = -2, 2) and columns (dk = -2, 2).
__constant__ unsigned char c_window_place[25] = {13, 17, 11, 18, 14, 21, 5, 3, 6, 23, 9, 1, 0, 2, 10, 22, 7, 4, 8, 24,
                                                 15, 19, 12, 20, 16};

// Eight lanes per new marker r: its quarter cell, the nearest of the markers in
// the 5x5 quarter cells around it, and the copy.  The reference visits the
// cells in that order and replaces the best by a strictly closer marker,
// so its result is the least distance (the rounded root) and, among equals, the
// first visited; the first of all where none is closer than the box is wide.
// The five cells of a window row are one run of the sorted list, which the lanes
// share.
//
// The lanes first look for the least distance between position codes, in FP32: a
// code is within one unit of the position, so a distance of codes is within
// 3 units (2 sqrt 2, in units of 2^-13 of the wider quarter cell) of the exact
// one, and a marker that is nearer than all others by 6 is the nearest.  Else
// (one window in 200, lattices, markers outside the quarter grid, boxes narrower
// than the distance) the squares are formed in FP64, and where another is within
// 8 units in the last place of the least the roots and places are compared.
//
// One thread per new marker followed some 100 dependent loads (list, then
// coordinates) one after the other, with few warps on the chip: 27 000 new
// markers 140 us, 1364 us a step at 1024 x 512.  The lanes with FP64 squares took
// 94 and 1086 us (the FP64 pipe), with the codes 44 and 405.
constexpr int RS_LANES = 8;

// By squared distances in FP64, for the group of lanes.
__device__ __noinline__ int exact_nearest(int nxl, double best, int kd, int lane, unsigned group,
                                          const int *__restrict__ qstart, const int *__restrict__ qsorted,
                                          const double *x, const double *z, double xn, double zn) {
    typedef unsigned long long u64;
    auto dist2 = [&](int j) {   // bits of the squared distance: they order like the value
        const double ax = xn - x[j], az = zn - z[j];
        return (u64)__double_as_longlong(__dadd_rn(__dmul_rn(ax, ax), __dmul_rn(az, az)));
    };
    u64 least = ~0ull, next = ~0ull;
    int m = -1;
    for (int w = 0; w < 5; w++)
        for (int s = qstart[kd + (w - 2) * nxl - 2] + lane; s < qstart[kd + (w - 2) * nxl + 3]; s += RS_LANES) {
            const int j = qsorted[s];
            const u64 d2 = dist2(j);
            if (d2 < least) { next = least; least = d2; m = j; }
            else if (d2 < next) next = d2;
        }
    u64 all = least;
    for (int o = 1; o < RS_LANES; o <<= 1) {
        const u64 v = __shfl_xor_sync(group, all, o);
        all = v < all ? v : all;
    }
    const double d = sqrt(__longlong_as_double((long long)all));
    const u64 near = all + 8;
    const bool closer = d < best;
    const unsigned mine = __ballot_sync(group, least <= near), more = __ballot_sync(group, next <= near);
    if (closer && more == 0 && __popc(mine) == 1) return __shfl_sync(group, m, __ffs(mine) - 1);
    // the first visited of the equally close (of all, if none is closer than the box is wide)
    u64 place = ~0ull;
    for (int w = 0; w < 5; w++)
        for (int c = 0; c < 5; c++) {
            const int b = qstart[kd + (w - 2) * nxl + c - 2], e = qstart[kd + (w - 2) * nxl + c - 1];
            for (int s = b + lane; s < e; s += RS_LANES) {
                const int j = qsorted[s];
                const u64 d2 = dist2(j);
                if (closer && (d2 > near || sqrt(__longlong_as_double((long long)d2)) != d)) continue;
                const u64 at = (u64)c_window_place[5 * w + c] << 32 | (unsigned)(s - b);
                if (at < place) { place = at; m = j; }
            }
        }
    u64 low = place;
    for (int o = 1; o < RS_LANES; o <<= 1) {
        const u64 v = __shfl_xor_sync(group, low, o);
        low = v < low ? v : low;
    }
    return __shfl_sync(group, m, __ffs(__ballot_sync(group, place == low)) - 1);
}

__global__ void k_reseed_write(quarter_geom q, mdz_dgrid g, int n, int nnew, int nreuse, const int *__restrict__ list,
                               const int *__restrict__ qstart, const int *__restrict__ qsorted,
                               const int *__restrict__ qcode, const int *__restrict__ inexact,
                               const int *__restrict__ reuse, double *x, double *z, int *phase, double *vx,
                               double *vz, mdz_attr_ptrs A, int direct, reseed_fields F) {
    const int wj = q.nzl - 4;
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int r = (int)(tid / RS_LANES), lane = threadIdx.x % RS_LANES;
    if (r >= nnew) return;   // whole groups of eight
    const unsigned group = 0xffu << (threadIdx.x & 24);
    const int qo = list[r];
    const int k = 2 + qo / wj, l = 2 + qo % wj, kd = k + l * q.nxl;
    const double xn = new_pos(q.xg0, k - 2, q.dx), zn = new_pos(q.zg0, l - 2, q.dz);
    int st[5], en[5];
#pragma unroll
    for (int w = 0; w < 5; w++) {
        st[w] = qstart[kd + (w - 2) * q.nxl - 2];
        en[w] = qstart[kd + (w - 2) * q.nxl + 3];
    }
    int m = -1;
    bool sure = false;
    if (!*inexact) {
        const int hx = (k << 13) + 4096, hz = (l << 13) + 4096;   // the centre of quarter cell (k, l)
        float least = INFINITY, next = INFINITY;
        int at = 0;
#pragma unroll
        for (int w = 0; w < 5; w++)
            for (int s = st[w] + lane; s < en[w]; s += RS_LANES) {
                const int c = qcode[s];
                const float ax = (float)(short)((c & 0xffff) - hx), az = (float)(short)((c >> 16) - hz);
                const float d2 = q.cx * ax * ax + q.cz * az * az;
                if (d2 < least) { next = least; least = d2; at = s; }
                else next = fminf(next, d2);
            }
        float all = least;
#pragma unroll
        for (int o = 1; o < RS_LANES; o <<= 1) all = fminf(all, __shfl_xor_sync(group, all, o));
        const float d = sqrtf(all), limit = (d + 6.001f) * (d + 6.001f) * 1.0001f;
        const unsigned mine = __ballot_sync(group, least <= limit), more = __ballot_sync(group, next <= limit);
        sure = more == 0 && __popc(mine) == 1 && (d + 3.001f) * 1.0001f < q.width;
        m = qsorted[at];
        m = __shfl_sync(group, m, __ffs(mine) - 1);
    }
    if (!sure) m = exact_nearest(q.nxl, q.xmax - q.xmin, kd, lane, group, qstart, qsorted, x, z, xn, zn);
    const int slot = r < nreuse ? reuse[r] : n + (r - nreuse);
    // the lanes take the properties between them
    if (lane == 5) { x[slot] = xn; z[slot] = zn; }
    if (lane == 6) { phase[slot] = phase[m]; vx[slot] = vx[m]; vz[slot] = vz[m]; }
    if (lane == 7) {
        A.a[MDZ_M_STRAIN][slot] = A.a[MDZ_M_STRAIN][m];
        A.a[MDZ_M_STRAIN_PL][slot] = A.a[MDZ_M_STRAIN_PL][m];
        A.a[MDZ_M_CMUL][slot] = A.a[MDZ_M_CMUL][m];
    }
    if (lane < 5) {
        double *a = A.a[MDZ_M_T];
        const double *f = F.T_n;
        if (lane == 1) { a = A.a[MDZ_M_P]; f = F.p_n; }
        if (lane == 2) { a = A.a[MDZ_M_SXXD]; f = F.sxxd_n; }
        if (lane == 3) { a = A.a[MDZ_M_SZZD]; f = F.szzd_n; }
        if (lane == 4) { a = A.a[MDZ_M_SXZ]; f = F.sxz_s; }
        a[slot] = direct ? a[m] : grid_to_new(g, xn, zn, lane == 4, f);
    }
}

// exclusive scan of in[0..n) into out[0..n] (out[n] = total), partial: scratch
static mdz_status scan_ints(mdz_ctx *ctx, int n, const int *in, int *out, int *partial, cudaStream_t st) {
    const int nb = (n + 1023) / 1024;
    k_scan_blocks<<<nb, 1024, 0, st>>>(n, in, out, partial);
    MDZ_LAUNCHED(ctx);
    k_scan_partials<<<1, 1024, 0, st>>>(nb, partial);
    MDZ_LAUNCHED(ctx);
    k_scan_add<<<nb, 1024, 0, st>>>(n, out, partial);
    MDZ_LAUNCHED(ctx);
    return MDZ_OK;
}

static mdz_status reseed_ws(mdz_ctx *ctx, const quarter_geom &q, mdz_reseed_ws *&W) {
    if (!ctx->reseed) ctx->reseed = new mdz_reseed_ws();
    W = ctx->reseed;
    const int nq = q.nxl * q.nzl, ni = (q.nxl - 4) * (q.nzl - 4);
    const long long cap = ctx->m.cap > 0 ? ctx->m.cap : 1;
    if (W->cap == cap && W->nq == nq) return MDZ_OK;
    mdz_reseed_free(ctx);
    ctx->reseed = W = new mdz_reseed_ws();
    auto A = [&](int *&p, long long cnt) { return cudaMalloc((void **)&p, sizeof(int) * (size_t)(cnt > 0 ? cnt : 1)); };
    MDZ_CUDA(ctx, A(W->qcell, cap));
    MDZ_CUDA(ctx, A(W->qsorted, cap));
    MDZ_CUDA(ctx, A(W->qcount, nq + 1));
    MDZ_CUDA(ctx, A(W->qstart, nq + 1));
    MDZ_CUDA(ctx, A(W->qpart, (nq + 1023) / 1024 + 1));
    MDZ_CUDA(ctx, A(W->flag, ni));
    MDZ_CUDA(ctx, A(W->rank, ni + 1));
    MDZ_CUDA(ctx, A(W->src, ni));   // list: quarter cell of each new marker
    MDZ_CUDA(ctx, A(W->ipart, (ni + 1023) / 1024 + 1));
    MDZ_CUDA(ctx, A(W->inact, cap));
    MDZ_CUDA(ctx, A(W->islot, cap + 1));
    MDZ_CUDA(ctx, A(W->reuse, cap));
    MDZ_CUDA(ctx, A(W->mpart, (cap + 1023) / 1024 + 1));
    MDZ_CUDA(ctx, A(W->status, 4));
    W->cap = cap;
    W->nq = nq;
    W->ni = ni;
    return MDZ_OK;
}

mdz_status mdz_dev_reseed(mdz_ctx *ctx, int min_part_cell, int direct, const double *T_n, const double *sxxd_n,
                          const double *szzd_n, const double *sxz_s, const double *p_n, cudaStream_t st,
                          int *n_added) {
    if (n_added) *n_added = 0;
    if (min_part_cell < 0) return mdz_fail(ctx, MDZ_ERR_ARG, "CountPartCell: min_part_cell < 0");
    if (!direct && (!T_n || !sxxd_n || !szzd_n || !sxz_s || !p_n))
        return mdz_fail(ctx, MDZ_ERR_ARG, "CountPartCell: DirectNeighbour = 0 needs T, sxxd, szzd, sxz and p");
    const quarter_geom q = make_quarter_geom(ctx);
    // quarter-cell indices are 32-bit: (2 Ncx + 4)(2 Ncz + 4) must stay below 2^31
    if ((long long)q.nxl * q.nzl > 2147483000LL)
        return mdz_fail(ctx, MDZ_ERR_UNSUPPORTED, "CountPartCell: %d x %d quarter cells exceed 2^31", q.nxl, q.nzl);
    mdz_reseed_ws *W = nullptr;
    mdz_status s = reseed_ws(ctx, q, W);
    if (s != MDZ_OK) return s;
    const int n = ctx->m.n, nq = W->nq, ni = W->ni;
    // quarter-cell bins, ascending marker index inside each
    int *const arrival = W->inact, *const code = W->islot;   // free until the inactive slots are listed
    int *const qcode = W->qcell;                             // free after the scatter
    MDZ_CUDA(ctx, cudaMemsetAsync(W->qcount, 0, sizeof(int) * (nq + 1), st));
    MDZ_CUDA(ctx, cudaMemsetAsync(W->status, 0, sizeof(int) * 4, st));
    if (n > 0) {
        k_quarter_count<<<mdz_blocks(n), MDZ_THREADS, 0, st>>>(n, ctx->m.x, ctx->m.z, ctx->m.phase, q, W->qcell,
                                                               code, arrival, W->qcount, W->status);
        MDZ_LAUNCHED(ctx);
    }
    if ((s = scan_ints(ctx, nq, W->qcount, W->qstart, W->qpart, st)) != MDZ_OK) return s;
    if (n > 0) {
        k_bin_scatter<<<mdz_blocks(n), MDZ_THREADS, 0, st>>>(n, W->qcell, arrival, W->qstart, W->qsorted);
        MDZ_LAUNCHED(ctx);
    }
    k_quarter_sort<<<mdz_blocks(nq), MDZ_THREADS, 0, st>>>(nq, W->qstart, W->qsorted, code, qcode);
    MDZ_LAUNCHED(ctx);
    // deficient quarter cells and their nearest markers, then the ranks
    const int thr = (int)(std::ceil((double)min_part_cell) / 4.0);
    k_reseed_cells<<<mdz_blocks(ni), MDZ_THREADS, 0, st>>>(q, ctx->g.BCp, W->qstart, thr, W->flag, W->status);
    MDZ_LAUNCHED(ctx);
    if ((s = scan_ints(ctx, ni, W->flag, W->rank, W->ipart, st)) != MDZ_OK) return s;
    k_reseed_list<<<mdz_blocks(ni), MDZ_THREADS, 0, st>>>(ni, W->flag, W->rank, W->src);
    MDZ_LAUNCHED(ctx);
    // inactive slots in index order
    int nreuse = 0;
    if (n > 0) {
        k_inactive_flags<<<mdz_blocks(n), MDZ_THREADS, 0, st>>>(n, ctx->m.phase, W->inact);
        MDZ_LAUNCHED(ctx);
        if ((s = scan_ints(ctx, n, W->inact, W->islot, W->mpart, st)) != MDZ_OK) return s;
        k_inactive_list<<<mdz_blocks(n), MDZ_THREADS, 0, st>>>(n, W->inact, W->islot, W->reuse);
        MDZ_LAUNCHED(ctx);
    }
    int h[3] = {0, 0, 0};
    MDZ_CUDA(ctx, cudaMemcpyAsync(&h[0], W->rank + ni, sizeof(int), cudaMemcpyDeviceToHost, st));
    if (n > 0) MDZ_CUDA(ctx, cudaMemcpyAsync(&h[1], W->islot + n, sizeof(int), cudaMemcpyDeviceToHost, st));
    MDZ_CUDA(ctx, cudaMemcpyAsync(&h[2], W->status, sizeof(int), cudaMemcpyDeviceToHost, st));
    MDZ_CUDA(ctx, cudaStreamSynchronize(st));
    const int nnew = h[0];
    nreuse = h[1];
    if (h[2]) return mdz_fail(ctx, MDZ_ERR_STATE, "CountPartCell: a quarter cell lacking markers has no marker within two quarter cells");
    const long long n_final = (long long)n + (nnew > nreuse ? nnew - nreuse : 0);
    if (n_final > ctx->m.cap)
        return mdz_fail(ctx, MDZ_ERR_CAPACITY, "CountPartCell: %lld markers after reseeding > capacity %lld", n_final,
                        ctx->m.cap);
    if (nnew > 0) {
        mdz_attr_ptrs A;
        for (int a = 0; a < MDZ_M_NATTR; a++) A.a[a] = ctx->m.attr[a];
        k_reseed_write<<<mdz_blocks((long long)nnew * RS_LANES), MDZ_THREADS, 0, st>>>(q, ctx->g, n, nnew, nreuse, W->src, W->qstart,
                                                                 W->qsorted, qcode, W->status + 1, W->reuse, ctx->m.x, ctx->m.z,
                                                                 ctx->m.phase, ctx->m.vx, ctx->m.vz, A, direct,
                                                                 reseed_fields{T_n, sxxd_n, szzd_n, sxz_s, p_n});
        MDZ_LAUNCHED(ctx);
    }
    ctx->m.n = (int)n_final;
    ctx->bins.valid = false;
    if (n_added) *n_added = nnew;
    return MDZ_OK;
}

extern "C" mdz_status mdz_CountPartCell(mdz_ctx *ctx, int reseed, int min_part_cell, int direct_neighbour,
                                        const double *T_n, const double *sxxd_n, const double *szzd_n,
                                        const double *sxz_s, const double *p_n, int *n_added) {
    if (!ctx) return MDZ_ERR_ARG;
    if (n_added) *n_added = 0;
    if (!reseed) return MDZ_OK;
    cudaStream_t st = ctx->stream;
    const mdz_dgrid &g = ctx->g;
    const size_t nc = (size_t)g.ncx * g.ncz, nv = (size_t)g.Nx * g.Nz;
    const double *d[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
    if (!direct_neighbour) {
        if (!T_n || !sxxd_n || !szzd_n || !sxz_s || !p_n)
            return mdz_fail(ctx, MDZ_ERR_ARG, "CountPartCell: DirectNeighbour = 0 needs T, sxxd, szzd, sxz and p");
        const double *hsrc[5] = {T_n, sxxd_n, szzd_n, sxz_s, p_n};
        static const int slot[5] = {0, 1, 2, 3, 6};   // staging slots (5 holds the time step's workspace)
        for (int i = 0; i < 5; i++) {
            const size_t cnt = i == 3 ? nv : nc;
            double *p = (double *)mdz_stage(ctx, slot[i], sizeof(double) * cnt);
            if (!p) return mdz_fail(ctx, MDZ_ERR_CUDA, "CountPartCell: staging allocation failed");
            MDZ_CUDA(ctx, cudaMemcpyAsync(p, hsrc[i], sizeof(double) * cnt, cudaMemcpyHostToDevice, st));
            d[i] = p;
        }
    }
    int added = 0;
    mdz_status s = mdz_dev_reseed(ctx, min_part_cell, direct_neighbour, d[0], d[1], d[2], d[3], d[4], st, &added);
    if (s != MDZ_OK) return s;
    MDZ_CUDA(ctx, cudaStreamSynchronize(st));
    if (n_added) *n_added = added;
    return MDZ_OK;
}
