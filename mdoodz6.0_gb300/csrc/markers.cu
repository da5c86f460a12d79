// Marker-side kernels: binning by cell and quadrant (counting sort), batched
// marker->grid projection as deterministic per-node sums, marker counts,
// grid->marker interpolation and RK4 advection.
//
// Reference behaviour followed (paths inside the MDOODZ 6.0 repository):
//   P2Mastah                  SOURCE/ParticleRoutines.c:3226-3537
//   CountPartCell_Old counts  SOURCE/ParticleRoutines.c:4485-4980
//   Interp_Grid2P             SOURCE/ParticleRoutines.c:2439-2608
//   Interp_Grid2P_centroids2  SOURCE/ParticleRoutines.c:2612-2862
//   V2P (TarasCorr = 0)       SOURCE/ParticleRoutines.c:60-252
//   RogerGuntherII / isoutPart SOURCE/AdvectionRoutines.c:569-628, 314-335
#include <cmath>
#include <cstring>
#include "mdz_internal.cuh"

// Nearest-node index along one line of a node set, as the reference computes
// it: ceil(d/h + 0.5) - 1 with d measured from the first line, clamped.
__device__ __forceinline__ int nearest_line(double x, double X0, double h, double ih, int n) {
    int i = quot_index(x - X0, h, ih, 0.5);
    i = i < 0 ? 0 : i;
    return i > n - 1 ? n - 1 : i;
}

// Lower-left cell index along one line (V2P / Interp_Grid2P): ceil(d/h) - 1.
__device__ __forceinline__ int lower_line(double x, double X0, double h, double ih) {
    return quot_index(x - X0, h, ih, 0.0);
}

// Two sets of lines with one spacing, and the distance of their first lines in
// 2^-20 of it (line_indices).
struct line_pair {
    const double *X, *Xh;
    double h, ih;
    long long off;
    int n;   // lines of the first set
};

static line_pair make_line_pair(const double *X, const double *Xh, double first, double first_h, double h, int n) {
    const double ih = 1.0 / h;
    return line_pair{X, Xh, h, ih, (long long)std::llround((first - first_h) * ih * 1048576.0), n};
}

// ---------------------------------------------------------------------------
// Binning: cell of each active marker = nearest centroid (the same formula and
// clamps as P2Mastah on centroids), and inside the cell the quadrant of its
// nearest vertex (the cell's corner (q & 1, q >> 1)): bin `quads` cell + q.  A
// cell is then the nearest-centroid list of its centroid and a quadrant a
// quarter of the nearest-vertex list of its corner, both contiguous.  quads is
// 1, without quadrants, where four times the cells leave 32 bits.
// cell[k]: the bin, arrival[k]: how many of the bin came before (in any order:
// the segments are sorted below), which saves the scatter its atomics.
// Bound by the FP64 pipe: four indices one by one took 135 us for 8.4 M markers,
// in pairs 85.
__device__ __forceinline__ void cell_and_side(const line_pair &L, double x, int &c, int &side) {
    int v;
    if (!line_indices(x - L.X[0], L.ih, 0.5, L.off, c, v)) {
        c = nearest_line(x, L.X[0], L.h, L.ih, L.n);
        v = nearest_line(x, L.Xh[0], L.h, L.ih, L.n + 1);
    }
    c = c < 0 ? 0 : (c > L.n - 1 ? L.n - 1 : c);
    v = v < 0 ? 0 : (v > L.n ? L.n : v);
    side = v > c;   // the vertex lines lie half a cell to either side of the centroid's
}

__global__ void k_bin_count(int n, const double *__restrict__ x, const double *__restrict__ z,
                            const int *__restrict__ phase, line_pair LX, line_pair LZ, int quads,
                            int *__restrict__ cell, int *__restrict__ arrival, int *__restrict__ count) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    if (phase[k] == -1) { cell[k] = -1; return; }
    int ic, jc, qx, qz;
    cell_and_side(LX, x[k], ic, qx);
    cell_and_side(LZ, z[k], jc, qz);
    int c = ic + jc * LX.n;
    if (quads == 4) c = 4 * c + qx + 2 * qz;
    cell[k] = c;
    arrival[k] = atomicAdd(&count[c], 1);
}

// Block-wise inclusive scan (1024 elements per block) of int counts; writes
// exclusive results to out[i+1] and block totals to partial[].
__global__ void k_scan_blocks(int n, const int *__restrict__ in, int *__restrict__ out, int *__restrict__ partial) {
    __shared__ int warp_sums[32];
    int i = blockIdx.x * 1024 + threadIdx.x;
    int v = i < n ? in[i] : 0;
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int s = v;
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += t;
    }
    if (lane == 31) warp_sums[wid] = s;
    __syncthreads();
    if (wid == 0) {
        int w = warp_sums[lane];
        for (int o = 1; o < 32; o <<= 1) {
            int t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        warp_sums[lane] = w;
    }
    __syncthreads();
    if (wid > 0) s += warp_sums[wid - 1];
    if (i < n) out[i + 1] = s;
    if (threadIdx.x == 1023) partial[blockIdx.x] = s;
}

// Serial-over-blocks scan of the block totals (one CTA; blocks <= a few thousand).
__global__ void k_scan_partials(int nb, int *partial) {
    __shared__ int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < nb; base += 1024) {
        int i = base + threadIdx.x;
        int v = i < nb ? partial[i] : 0;
        // inclusive scan across the CTA, simple two-level
        __shared__ int buf[1024];
        buf[threadIdx.x] = v;
        __syncthreads();
        for (int o = 1; o < 1024; o <<= 1) {
            int t = threadIdx.x >= o ? buf[threadIdx.x - o] : 0;
            __syncthreads();
            buf[threadIdx.x] += t;
            __syncthreads();
        }
        int excl = buf[threadIdx.x] - v + carry;
        __syncthreads();
        if (i < nb) partial[i] = excl;
        if (threadIdx.x == 1023) carry += buf[1023];
        __syncthreads();
    }
}

__global__ void k_scan_add(int n, int *__restrict__ out, const int *__restrict__ partial) {
    int i = blockIdx.x * 1024 + threadIdx.x;
    if (i == 0) out[0] = 0;
    if (i < n) out[i + 1] += partial[blockIdx.x];
}

__global__ void k_bin_scatter(int n, const int *__restrict__ cell, const int *__restrict__ arrival,
                              const int *__restrict__ start, int *__restrict__ sorted) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    int c = cell[k];
    if (c >= 0) sorted[start[c] + arrival[k]] = k;
}

// Make the order inside each bin ascending in marker index, so that every
// projection sums in a fixed order (bit-reproducible run to run).
__global__ void k_bin_sort_segments(int ncells, const int *__restrict__ start, int *__restrict__ sorted) {
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncells) return;
    int b = start[c], e = start[c + 1];
    for (int i = b + 1; i < e; i++) {
        int v = sorted[i], j = i - 1;
        while (j >= b && sorted[j] > v) { sorted[j + 1] = sorted[j]; j--; }
        sorted[j + 1] = v;
    }
}

mdz_status mdz_ensure_bins(mdz_ctx *ctx, cudaStream_t st) {
    mdz_bins &B = ctx->bins;
    if (B.valid) return MDZ_OK;
    const mdz_dgrid &g = ctx->g;
    const int n = ctx->m.n, nb = B.quads * B.ncells;
    MDZ_CUDA(ctx, cudaMemsetAsync(B.count, 0, sizeof(int) * ((size_t)nb + 1), st));
    if (n > 0) {
        const mdz_grid_desc &hd = ctx->host_desc;
        k_bin_count<<<mdz_blocks(n), MDZ_THREADS, 0, st>>>(n, ctx->m.x, ctx->m.z, ctx->m.phase,
                                                           make_line_pair(g.xc, g.xg, hd.xc[0], hd.xg[0], g.dx, g.ncx),
                                                           make_line_pair(g.zc, g.zg, hd.zc[0], hd.zg[0], g.dz, g.ncz),
                                                           B.quads, B.cell, B.arrival, B.count);
        MDZ_LAUNCHED(ctx);
    }
    const int blocks = (int)(((size_t)nb + 1023) / 1024);
    k_scan_blocks<<<blocks, 1024, 0, st>>>(nb, B.count, B.start, B.scan_partials);
    MDZ_LAUNCHED(ctx);
    k_scan_partials<<<1, 1024, 0, st>>>(blocks, B.scan_partials);
    MDZ_LAUNCHED(ctx);
    k_scan_add<<<blocks, 1024, 0, st>>>(nb, B.start, B.scan_partials);
    MDZ_LAUNCHED(ctx);
    if (n > 0) {
        k_bin_scatter<<<mdz_blocks(n), MDZ_THREADS, 0, st>>>(n, B.cell, B.arrival, B.start, B.sorted);
        MDZ_LAUNCHED(ctx);
    }
    k_bin_sort_segments<<<mdz_blocks(nb), MDZ_THREADS, 0, st>>>(nb, B.start, B.sorted);
    MDZ_LAUNCHED(ctx);
    B.valid = true;
    return MDZ_OK;
}

// ---------------------------------------------------------------------------
// Batched projection.  Every node gathers, from the markers of the cells that
// can hold its contributors, exactly the tent weights P2Mastah scatters: each marker finds its nearest node (ip, jp) with the reference's
// formula and clamps, then contributes to (ip, jp) and, for the 9-cell
// stencil, to the 8 neighbours, with distances measured from X[ip] +/- dx.
struct p2g_fields {
    const double *val[MDZ_P2G_MAX_FIELDS];   // per-marker values, or per-phase table
    int per_phase[MDZ_P2G_MAX_FIELDS];       // 1: val is indexed by phase (flag 0)
    int avg[MDZ_P2G_MAX_FIELDS];
    double *out[MDZ_P2G_MAX_FIELDS];
    int *empty;   // when set, counts active nodes that received no marker weight (phase fractions only)
};

// Candidate cell range along one direction for node i of a node set whose
// lines are of kind `kind` (0: centroid lines, 1: vertex lines, 2: ghosted lines).
__device__ __forceinline__ void cell_range(int i, int h, int kind, int n_nodes, int n_cells, int &lo, int &hi) {
    lo = i - h - kind;
    hi = i + h;
    if (i - h <= 0) lo = 0;
    if (i + h >= n_nodes - 1) hi = n_cells - 1;
    lo = lo < 0 ? 0 : lo;
    hi = hi > n_cells - 1 ? n_cells - 1 : hi;
}

// Node value B / W by the reciprocal of W that the node's fields share: one step
// on the remainder makes the quotient the rounded one but for rare last bits
// (Markstein, IBM J. Res. Dev. 34, 1990), in 3 FP64 instructions.
__device__ __forceinline__ double over_weight(double B, double W, double rW) {
    const double q = B * rW;
    const unsigned e = ((unsigned)__double2hiint(q) >> 20) & 0x7ffu;   // biased exponent: 0 for a zero, 2^-900 .. 2^900
    if ((e < 123u || e > 1923u) && (__double_as_longlong(B) << 1) != 0) return B / W;
    return __fma_rn(__fma_rn(-q, W, B), rW, q);
}

template <int NF, int NPH>
__device__ __forceinline__ void p2g_finish(int node, int nn, signed char tag, double Wm, const double *BmWm,
                                           const double *Wph, const p2g_fields &F, int nph_rt,
                                           double *__restrict__ phase_perc) {
    const bool air = tag == 30 || tag == 31;
    const bool skip = fabs(Wm) < 1e-30 || air;
    if (F.empty && phase_perc && !air && fabs(Wm) < 1e-30) atomicAdd(F.empty, 1);
    const double rW = 1.0 / Wm;
#pragma unroll
    for (int f = 0; f < NF; f++) {
        if (skip) continue;
        double v = over_weight(BmWm[f], Wm, rW);
        if (F.avg[f] == 1) v = 1.0 / v;
        if (F.avg[f] == 2) v = exp(v);
        F.out[f][node] = v;
    }
    if (phase_perc) {
#pragma unroll
        for (int p = 0; p < NPH; p++)
            if (p < nph_rt) phase_perc[(size_t)p * nn + node] = skip ? Wph[p] : over_weight(Wph[p], Wm, rW);
    }
}

template <int NF, int NPH>
__global__ void __launch_bounds__(128) k_p2g_gather(
    int nnx, int nnz, const double *__restrict__ X, const double *__restrict__ Z, const signed char *__restrict__ tag,
    int kindx, int kindz, int h, double dx, double dz, double idx, double idz, double idxi, double idzi, int ncx,
    int ncz, int quads, const int *__restrict__ start, const int *__restrict__ sorted, const double *__restrict__ mx, const double *__restrict__ mz, const int *__restrict__ mphase, p2g_fields F,
    int nph_rt, double *__restrict__ phase_perc) {
    int node = blockIdx.x * blockDim.x + threadIdx.x;
    if (node >= nnx * nnz) return;
    int i = node % nnx, j = node / nnx;
    int clo, chi, rlo, rhi;
    cell_range(i, h, kindx, nnx, ncx, clo, chi);
    cell_range(j, h, kindz, nnz, ncz, rlo, rhi);
    double Wm = 0.0, BmWm[NF > 0 ? NF : 1], Wph[NPH > 0 ? NPH : 1];
#pragma unroll
    for (int f = 0; f < NF; f++) BmWm[f] = 0.0;
#pragma unroll
    for (int p = 0; p < NPH; p++) Wph[p] = 0.0;
    const double X0 = X[0], Z0 = Z[0];
    // (1/dx, 1/dz and the reciprocal interpolation widths come from the host:
    // an FP64 division per thread is a long instruction sequence on this part)
    // contribution of marker k, whose nearest node (ip, jp) is within h of this one
    auto add = [&](int k, int ip, int jp, int di, int dj) {
        const double xk = mx[k], zk = mz[k];
        double Xn = X[ip], Zn = Z[jp];
        if (di > 0) Xn = X[ip] + dx;
        if (di < 0) Xn = X[ip] - dx;
        if (dj > 0) Zn = Z[jp] + dz;
        if (dj < 0) Zn = Z[jp] - dz;
        double dxm = fabs(Xn - xk), dzm = fabs(Zn - zk);
        double w = (1.0 - dxm * idxi) * (1.0 - dzm * idzi);
        int p = mphase[k];
        Wm += w;
#pragma unroll
        for (int pp = 0; pp < NPH; pp++)
            if (p == pp) Wph[pp] += w;
#pragma unroll
        for (int f = 0; f < NF; f++) {
            double v = F.per_phase[f] ? F.val[f][p] : F.val[f][k];
            if (F.avg[f] == 1) v = 1.0 / v;
            if (F.avg[f] == 2) v = log(v);
            BmWm[f] += v * w;
        }
    };
    // Markers by cell rows upwards, cells left to right, bins in order inside a cell.
    for (int r = rlo; r <= rhi; r++) {
        const size_t b = start[(size_t)quads * (clo + r * ncx)], e = start[(size_t)quads * (chi + r * ncx + 1)];
        for (size_t q = b; q < e; q++) {
            const int k = sorted[q];
            const int ip = nearest_line(mx[k], X0, dx, idx, nnx), jp = nearest_line(mz[k], Z0, dz, idz, nnz);
            int di = i - ip, dj = j - jp;
            if (di < -h || di > h || dj < -h || dj > h) continue;
            add(k, ip, jp, di, dj);
        }
    }
    p2g_finish<NF, NPH>(node, nnx * nnz, tag[node], Wm, BmWm, Wph, F, nph_rt, phase_perc);
}

// Projection on centroids or vertices, whose nearest-node lists are contiguous
// runs of the bins (one per centroid, one per quadrant around a vertex).  A CTA
// has 4 rows of 32 nodes; the markers of the nodes and, for the nine-cell
// stencil (H = 1), of the ring of nodes around them go through shared memory
// four per owner node at a time: read by four neighbouring lanes per owner (a
// full 32-byte sector where the markers lie in bin order), transformed once
// (reciprocal, logarithm), and summed by one lane per node.
//
// With a thread per node reading its markers from global memory a load
// touched 32 sectors for 32 values and, with more nodes in flight than L1 has
// sectors for, most markers came from L2 several times; vertices tested every
// marker of their candidate cells (four for one that counts, 16 for nine), and
// the nine-cell stencil took reciprocals and logarithms nine times per marker.
// Four markers per owner at a time: with two or eight the six-field centroid
// projection takes 2.4 and 1.4 times as long (half sectors; two CTAs per SM).
// Now bound by the FP64 pipe (72 % active; 20 instructions a marker): 8.4 M
// markers onto 1024 x 512 centroids, six fields and four phases, 1249 -> 350 us;
// 1.1 M onto 302 x 151 vertices, nine cells, three harmonic means, 945 -> 311 us.
constexpr int P2G_W = 32, P2G_R = 4, P2G_LEN = 4, P2G_PAD = 5;   // padded owner: no bank conflicts in the sums

template <int NF, int H>
constexpr size_t p2g_tile_bytes() {
    return (size_t)(P2G_W + 2 * H) * (P2G_R + 2 * H) * (P2G_PAD * ((2 + NF) * 8 + 4) + 8 * 4);
}

template <int NF, int NPH, int H>
__global__ void __launch_bounds__(P2G_W *P2G_R) k_p2g_tile(
    int nnx, int nnz, int vert, const double *__restrict__ X, const double *__restrict__ Z,
    const signed char *__restrict__ tag, double dx, double dz, double idxi, double idzi, int ncx, int ncz,
    const int *__restrict__ start, const int *__restrict__ sorted, const double *__restrict__ mx,
    const double *__restrict__ mz, const int *__restrict__ mphase, p2g_fields F, int nph_rt,
    double *__restrict__ phase_perc) {
    constexpr int OW = P2G_W + 2 * H, OR = P2G_R + 2 * H, NO = OW * OR;
    constexpr int NONE = -2147483647 - 1;   // no marker in this place
    extern __shared__ double sm[];
    double *sx = sm, *sz = sx + NO * P2G_PAD, *sv = sz + NO * P2G_PAD;
    int *sp = (int *)(sv + NF * NO * P2G_PAD), *run = sp + NO * P2G_PAD, *end = run + 4 * NO;
    const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
    const int tiles = (nnx + P2G_W - 1) / P2G_W;
    const int i0 = (blockIdx.x % tiles) * P2G_W, j0 = (blockIdx.x / tiles) * P2G_R;
    // H = 0: the owners of a row are its own nodes, and a warp needs no other
    const int o_lo = H ? threadIdx.x : row * OW + lane, o_hi = H ? NO : row * OW + OW;
    const int o_step = H ? P2G_W * P2G_R : 32;
    auto meet = [&]() {
        if (H) __syncthreads();
        else __syncwarp();
    };
    // runs of the owners: marker m of owner o is sorted[run[r][o] + m], r the run with m < end[r][o]
    int longest = 0;
    for (int o = o_lo; o < o_hi; o += o_step) {
        const int i = i0 + o % OW - H, j = j0 + o / OW - H;
        const bool in = i >= 0 && i < nnx && j >= 0 && j < nnz;
        int len = 0;
#pragma unroll
        for (int r = 0; r < 4; r++) {
            int b = 0, e = 0;
            if (in && vert) {
                const int ci = i - 1 + (r & 1), cj = j - 1 + (r >> 1);
                if (ci >= 0 && ci < ncx && cj >= 0 && cj < ncz) {
                    const size_t q = 4 * (size_t)(ci + cj * ncx) + 3 - r;
                    b = start[q];
                    e = start[q + 1];
                }
            } else if (in && r == 0) {
                const size_t q = 4 * (size_t)(i + j * ncx);
                b = start[q];
                e = start[q + 4];
            }
            run[r * NO + o] = b - len;
            len += e - b;
            end[r * NO + o] = len;
        }
        longest = len > longest ? len : longest;
    }
    longest = __reduce_max_sync(0xffffffffu, longest);
    if (H) {
        __shared__ int s_longest[P2G_R];
        if (lane == 0) s_longest[row] = longest;
        __syncthreads();
        for (int w = 0; w < P2G_R; w++) longest = s_longest[w] > longest ? s_longest[w] : longest;
    }
    const int i = i0 + lane, j = j0 + row;
    const bool valid = i < nnx && j < nnz;
    // coordinates of the node, and of its owners' lines seen from there: X[ip] +- dx
    double Xn[2 * H + 1], Zn[2 * H + 1];
#pragma unroll
    for (int d = -H; d <= H; d++) {
        const int ip = i - d, jp = j - d;   // owner at distance d
        Xn[d + H] = ip >= 0 && ip < nnx ? (d > 0 ? X[ip] + dx : d < 0 ? X[ip] - dx : X[ip]) : 0.0;
        Zn[d + H] = jp >= 0 && jp < nnz ? (d > 0 ? Z[jp] + dz : d < 0 ? Z[jp] - dz : Z[jp]) : 0.0;
    }
    double Wm = 0.0, BmWm[NF > 0 ? NF : 1], Wph[NPH > 0 ? NPH : 1];
#pragma unroll
    for (int f = 0; f < NF; f++) BmWm[f] = 0.0;
#pragma unroll
    for (int p = 0; p < NPH; p++) Wph[p] = 0.0;
    for (int t = 0; t < longest; t += P2G_LEN) {
        meet();
        // four places per lane at a time, so that their loads are in flight together
        const int s_hi = o_hi * P2G_LEN;
        for (int s0 = H ? (int)threadIdx.x : row * OW * P2G_LEN + lane; s0 < s_hi; s0 += 4 * o_step) {
            int k[4], p[4], at[4];
            double a[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int s = s0 + u * o_step, o = s / P2G_LEN, m = t + s % P2G_LEN;
                at[u] = s < s_hi ? o * P2G_PAD + s % P2G_LEN : -1;
                k[u] = -1;
                p[u] = NONE;
                if (s < s_hi && m < end[3 * NO + o]) {
                    int r = 0;
                    if (vert) r = (m >= end[o]) + (m >= end[NO + o]) + (m >= end[2 * NO + o]);
                    k[u] = sorted[run[r * NO + o] + m];
                }
            }
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (k[u] >= 0) p[u] = mphase[k[u]];
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (at[u] >= 0) sp[at[u]] = p[u];
#pragma unroll
            for (int f = -2; f < NF; f++) {
                const double *src = f == -2 ? mx : f == -1 ? mz : F.val[f < 0 ? 0 : f];
                const bool per_phase = f >= 0 && F.per_phase[f < 0 ? 0 : f];
                const int avg = f >= 0 ? F.avg[f < 0 ? 0 : f] : 0;
#pragma unroll
                for (int u = 0; u < 4; u++) a[u] = k[u] >= 0 ? src[per_phase ? p[u] : k[u]] : 1.0;
                if (avg == 1) {
#pragma unroll
                    for (int u = 0; u < 4; u++) a[u] = 1.0 / a[u];
                } else if (avg == 2) {
#pragma unroll
                    for (int u = 0; u < 4; u++) a[u] = log(a[u]);
                }
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (k[u] >= 0) sm[(f + 2) * NO * P2G_PAD + at[u]] = a[u];
            }
        }
        meet();
        if (!valid) continue;
#pragma unroll
        for (int dj = H; dj >= -H; dj--) {   // owner rows upwards, owners left to right
#pragma unroll
            for (int di = H; di >= -H; di--) {
                const int o = (row + H - dj) * OW + lane + H - di;
#pragma unroll
                for (int m = 0; m < P2G_LEN; m++) {
                    const int at = o * P2G_PAD + m, p = sp[at];
                    if (p == NONE) break;
                    const double dxm = fabs(Xn[di + H] - sx[at]), dzm = fabs(Zn[dj + H] - sz[at]);
                    const double w = (1.0 - dxm * idxi) * (1.0 - dzm * idzi);
                    Wm += w;
#pragma unroll
                    for (int pp = 0; pp < NPH; pp++)
                        if (p == pp) Wph[pp] += w;
#pragma unroll
                    for (int f = 0; f < NF; f++) BmWm[f] += sv[f * NO * P2G_PAD + at] * w;
                }
            }
        }
    }
    if (valid) {
        const int node = i + j * nnx;
        p2g_finish<NF, NPH>(node, nnx * nnz, tag[node], Wm, BmWm, Wph, F, nph_rt, phase_perc);
    }
}

template <int NF, int NPH, int H>
static cudaError_t launch_p2g_tile(int vert, cudaStream_t st, const mdz_nodeset &ns, double dxi, double dzi,
                                   const mdz_ctx *ctx, const p2g_fields &F, int nph, double *pp) {
    const mdz_dgrid &g = ctx->g;
    const long long tiles = (long long)((ns.nx + P2G_W - 1) / P2G_W) * ((ns.nz + P2G_R - 1) / P2G_R);
    const size_t bytes = p2g_tile_bytes<NF, H>();
    cudaError_t e = cudaFuncSetAttribute(k_p2g_tile<NF, NPH, H>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    k_p2g_tile<NF, NPH, H><<<(unsigned)tiles, P2G_W * P2G_R, bytes, st>>>(
        ns.nx, ns.nz, vert, ns.X, ns.Z, ns.tag, g.dx, g.dz, 1.0 / dxi, 1.0 / dzi, g.ncx, g.ncz, ctx->bins.start,
        ctx->bins.sorted, ctx->m.x, ctx->m.z, ctx->m.phase, F, nph, pp);
    return cudaSuccess;
}

template <int NF, int NPH>
static cudaError_t launch_p2g(int kx, int kz, int h, cudaStream_t st, const mdz_nodeset &ns, double dxi, double dzi,
                              const mdz_ctx *ctx, const p2g_fields &F, int nph, double *pp) {
    const mdz_dgrid &g = ctx->g;
    const mdz_bins &B = ctx->bins;
    // centroids and vertices with quadrant bins; velocity nodes have one line of either kind
    if (B.quads == 4 && kx == kz)
        return h ? launch_p2g_tile<NF, NPH, 1>(kx, st, ns, dxi, dzi, ctx, F, nph, pp)
                 : launch_p2g_tile<NF, NPH, 0>(kx, st, ns, dxi, dzi, ctx, F, nph, pp);
    k_p2g_gather<NF, NPH><<<mdz_blocks(ns.nx * ns.nz, 128), 128, 0, st>>>(
        ns.nx, ns.nz, ns.X, ns.Z, ns.tag, kx, kz, h, g.dx, g.dz, 1.0 / g.dx, 1.0 / g.dz, 1.0 / dxi, 1.0 / dzi, g.ncx,
        g.ncz, B.quads, B.start, B.sorted, ctx->m.x, ctx->m.z, ctx->m.phase, F, nph, pp);
    return cudaSuccess;
}

template <int NF>
static cudaError_t launch_p2g_nf(int nph, int kx, int kz, int h, cudaStream_t st, const mdz_nodeset &ns, double dxi,
                                 double dzi, const mdz_ctx *ctx, const p2g_fields &F, double *pp) {
    if (pp == nullptr || nph <= 0) return launch_p2g<NF, 0>(kx, kz, h, st, ns, dxi, dzi, ctx, F, 0, nullptr);
    if (nph <= 4) return launch_p2g<NF, 4>(kx, kz, h, st, ns, dxi, dzi, ctx, F, nph, pp);
    return launch_p2g<NF, MDZ_MAX_PHASES>(kx, kz, h, st, ns, dxi, dzi, ctx, F, nph, pp);
}

// Core projection on the resident markers (device pointers everywhere).
static mdz_status p2g_core(mdz_ctx *ctx, const p2g_fields &F, int nf, double *d_phase_perc, int centroid,
                           int itp_stencil, cudaStream_t st) {
    if (itp_stencil != 1 && itp_stencil != 9)
        return mdz_fail(ctx, MDZ_ERR_ARG, "P2G: itp_stencil must be 1 or 9 (got %d)", itp_stencil);
    if (centroid < -2 || centroid > 1) return mdz_fail(ctx, MDZ_ERR_ARG, "P2G: bad node set %d", centroid);
    if (nf < 0 || nf > MDZ_P2G_MAX_FIELDS) return mdz_fail(ctx, MDZ_ERR_ARG, "P2G: too many fields (%d)", nf);
    mdz_status s = mdz_ensure_bins(ctx, st);
    if (s != MDZ_OK) return s;
    const mdz_dgrid &g = ctx->g;
    mdz_nodeset ns = mdz_get_nodeset(ctx, centroid);
    int kx = centroid == MDZ_NODES_CENTROIDS ? 0 : (centroid == MDZ_NODES_VZ ? 2 : 1);
    int kz = centroid == MDZ_NODES_CENTROIDS ? 0 : (centroid == MDZ_NODES_VX ? 2 : 1);
    int h = itp_stencil == 9 ? 1 : 0;
    double dxi = itp_stencil == 9 ? 3.0 * g.dx / 2.0 : g.dx / 2.0;
    double dzi = itp_stencil == 9 ? 3.0 * g.dz / 2.0 : g.dz / 2.0;
    int nn = ns.nx * ns.nz;
    int nph = d_phase_perc ? ctx->n_phases : 0;
    p2g_fields Fc = F;
    Fc.empty = d_phase_perc ? ctx->p2g_empty : nullptr;
    cudaEvent_t ev;
    mdz_prof_begin(ctx, MDZ_PROF_P2G, st, &ev);
    switch (nf) {
#define CASE(N) case N: MDZ_CUDA(ctx, launch_p2g_nf<N>(nph, kx, kz, h, st, ns, dxi, dzi, ctx, Fc, d_phase_perc)); break;
        CASE(0) CASE(1) CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(7) CASE(8)
#undef CASE
    }
    MDZ_LAUNCHED(ctx);
    {   // algorithmic bytes: each marker's position, phase and per-marker
        // fields read once; each node's fields and phase fractions written once
        int nfm = 0;
        for (int f = 0; f < nf; f++) nfm += F.per_phase[f] ? 0 : 1;
        const double bytes = (double)ctx->m.n * (20.0 + 8.0 * nfm) + 8.0 * (double)nn * (nf + nph);
        mdz_prof_end(ctx, MDZ_PROF_P2G, bytes, st, ev);
    }
    return MDZ_OK;
}

extern "C" mdz_status mdz_dev_p2g(mdz_ctx *ctx, int n_fields, const double *const *d_values, const int *avg,
                                  double *const *d_out, double *d_phase_perc, int centroid, int itp_stencil,
                                  void *stream) {
    if (!ctx) return MDZ_ERR_ARG;
    if (n_fields < 0 || n_fields > MDZ_P2G_MAX_FIELDS || (n_fields > 0 && (!d_values || !avg || !d_out)))
        return mdz_fail(ctx, MDZ_ERR_ARG, "mdz_dev_p2g: bad field arguments");
    if (d_phase_perc && centroid != MDZ_NODES_CENTROIDS && centroid != MDZ_NODES_VERTICES)
        return mdz_fail(ctx, MDZ_ERR_ARG, "mdz_dev_p2g: phase fractions exist on centroids and vertices only");
    p2g_fields F{};
    for (int f = 0; f < n_fields; f++) {
        if (avg[f] < 0 || avg[f] > 2) return mdz_fail(ctx, MDZ_ERR_ARG, "mdz_dev_p2g: avg must be 0, 1 or 2");
        F.val[f] = d_values[f]; F.per_phase[f] = 0; F.avg[f] = avg[f]; F.out[f] = d_out[f];
    }
    cudaStream_t st = stream ? (cudaStream_t)stream : ctx->stream;
    return p2g_core(ctx, F, n_fields, d_phase_perc, centroid, itp_stencil, st);
}

extern "C" mdz_status mdz_P2Mastah(mdz_ctx *ctx, const double *mat_prop, double *node_field,
                                   const signed char *node_type, int flag, int avg, int prop, int centroid,
                                   int itp_stencil, double *phase_perc) {
    if (!ctx) return MDZ_ERR_ARG;
    if (centroid < -2 || centroid > 1) return mdz_fail(ctx, MDZ_ERR_ARG, "P2Mastah: bad node set %d", centroid);
    if (flag != 0 && flag != 1) return mdz_fail(ctx, MDZ_ERR_ARG, "P2Mastah: flag must be 0 or 1");
    if (avg < 0 || avg > 2) return mdz_fail(ctx, MDZ_ERR_ARG, "P2Mastah: avg must be 0, 1 or 2");
    if (prop == 1 && (!phase_perc || (centroid != 0 && centroid != 1)))
        return mdz_fail(ctx, MDZ_ERR_ARG, "P2Mastah: prop=1 needs phase_perc on centroids or vertices");
    if (prop == 0 && (!mat_prop || !node_field)) return mdz_fail(ctx, MDZ_ERR_ARG, "P2Mastah: null field pointers");
    cudaStream_t st = ctx->stream;
    mdz_nodeset ns = mdz_get_nodeset(ctx, centroid);
    size_t nn = (size_t)ns.nx * ns.nz;
    int n = ctx->m.n;
    // node tags: the caller's array decides which nodes are skipped
    signed char *dtag = nullptr;
    if (node_type) {
        dtag = (signed char *)mdz_stage(ctx, 3, nn);
        if (!dtag) return mdz_fail(ctx, MDZ_ERR_CUDA, "P2Mastah: staging allocation failed");
        MDZ_CUDA(ctx, cudaMemcpyAsync(dtag, node_type, nn, cudaMemcpyHostToDevice, st));
    }
    p2g_fields F{};
    int nf = 0;
    double *dout = nullptr, *dpp = nullptr;
    if (prop == 0) {
        size_t nval = flag == 0 ? (size_t)ctx->n_phases : (size_t)n;
        double *dval = (double *)mdz_stage(ctx, 0, sizeof(double) * (nval ? nval : 1));
        dout = (double *)mdz_stage(ctx, 1, sizeof(double) * nn);
        if (!dval || !dout) return mdz_fail(ctx, MDZ_ERR_CUDA, "P2Mastah: staging allocation failed");
        if (nval) MDZ_CUDA(ctx, cudaMemcpyAsync(dval, mat_prop, sizeof(double) * nval, cudaMemcpyHostToDevice, st));
        MDZ_CUDA(ctx, cudaMemcpyAsync(dout, node_field, sizeof(double) * nn, cudaMemcpyHostToDevice, st));
        F.val[0] = dval; F.per_phase[0] = flag == 0; F.avg[0] = avg; F.out[0] = dout;
        nf = 1;
    } else {
        dpp = (double *)mdz_stage(ctx, 2, sizeof(double) * nn * ctx->n_phases);
        if (!dpp) return mdz_fail(ctx, MDZ_ERR_CUDA, "P2Mastah: staging allocation failed");
    }
    // swap in the caller's tags for this call
    mdz_dgrid saved = ctx->g;
    if (dtag) {
        if (centroid == 1) ctx->g.BCp = dtag;
        else if (centroid == 0) ctx->g.BCg = dtag;
        else if (centroid == -1) ctx->g.BCu = dtag;
        else ctx->g.BCv = dtag;
    }
    mdz_status s = p2g_core(ctx, F, nf, dpp, centroid, itp_stencil, st);
    ctx->g = saved;
    if (s != MDZ_OK) return s;
    if (prop == 0) MDZ_CUDA(ctx, cudaMemcpyAsync(node_field, dout, sizeof(double) * nn, cudaMemcpyDeviceToHost, st));
    else MDZ_CUDA(ctx, cudaMemcpyAsync(phase_perc, dpp, sizeof(double) * nn * ctx->n_phases, cudaMemcpyDeviceToHost, st));
    MDZ_CUDA(ctx, cudaStreamSynchronize(st));
    return MDZ_OK;
}

// ---------------------------------------------------------------------------
// Counts per cell / vertex and per (node, phase): integer, exact.
template <int NPH>
__global__ void k_count_nodes(int nnx, int nnz, int kindx, int kindz, const double *__restrict__ X,
                              const double *__restrict__ Z, double dx, double dz, int ncx, int ncz, int quads,
                              const int *__restrict__ start, const int *__restrict__ sorted,
                              const double *__restrict__ mx, const double *__restrict__ mz,
                              const int *__restrict__ mphase, int nph, int *__restrict__ count,
                              int *__restrict__ phase_count) {
    int node = blockIdx.x * blockDim.x + threadIdx.x;
    if (node >= nnx * nnz) return;
    int i = node % nnx, j = node / nnx;
    int clo, chi, rlo, rhi;
    cell_range(i, 0, kindx, nnx, ncx, clo, chi);
    cell_range(j, 0, kindz, nnz, ncz, rlo, rhi);
    int cnt = 0, pc[NPH];
#pragma unroll
    for (int p = 0; p < NPH; p++) pc[p] = 0;
    for (int r = rlo; r <= rhi; r++) {
        int b = start[(size_t)quads * (clo + r * ncx)], e = start[(size_t)quads * (chi + r * ncx + 1)];
        for (int q = b; q < e; q++) {
            int k = sorted[q];
            if (nearest_line(mx[k], X[0], dx, 1.0 / dx, nnx) != i || nearest_line(mz[k], Z[0], dz, 1.0 / dz, nnz) != j)
                continue;
            int p = mphase[k];
            if (p < 0) continue;
            cnt++;
#pragma unroll
            for (int pp = 0; pp < NPH; pp++)
                if (p == pp) pc[pp]++;
        }
    }
    if (count) count[node] = cnt;
    if (phase_count) {
        int nn = nnx * nnz;
#pragma unroll
        for (int p = 0; p < NPH; p++)
            if (p < nph) phase_count[(size_t)p * nn + node] = pc[p];
    }
}

extern "C" mdz_status mdz_count_markers(mdz_ctx *ctx, int *nb_part_cell, int *nb_part_vert, int *phase_count_cell,
                                        int *phase_count_vert) {
    if (!ctx) return MDZ_ERR_ARG;
    cudaStream_t st = ctx->stream;
    mdz_status s = mdz_ensure_bins(ctx, st);
    if (s != MDZ_OK) return s;
    const mdz_dgrid &g = ctx->g;
    for (int which = 0; which < 2; which++) {
        int *hc = which ? nb_part_vert : nb_part_cell;
        int *hp = which ? phase_count_vert : phase_count_cell;
        if (!hc && !hp) continue;
        int centroid = which ? MDZ_NODES_VERTICES : MDZ_NODES_CENTROIDS;
        mdz_nodeset ns = mdz_get_nodeset(ctx, centroid);
        int nn = ns.nx * ns.nz, kind = which ? 1 : 0;
        int *dc = (int *)mdz_stage(ctx, 4, sizeof(int) * nn);
        int *dp = (int *)mdz_stage(ctx, 5, sizeof(int) * (size_t)nn * ctx->n_phases);
        if (!dc || !dp) return mdz_fail(ctx, MDZ_ERR_CUDA, "count: staging allocation failed");
        if (ctx->n_phases <= 4)
            k_count_nodes<4><<<mdz_blocks(nn), MDZ_THREADS, 0, st>>>(ns.nx, ns.nz, kind, kind, ns.X, ns.Z, g.dx, g.dz,
                                                                    g.ncx, g.ncz, ctx->bins.quads, ctx->bins.start,
                                                                    ctx->bins.sorted, ctx->m.x, ctx->m.z, ctx->m.phase, ctx->n_phases,
                                                                    dc, dp);
        else
            k_count_nodes<MDZ_MAX_PHASES><<<mdz_blocks(nn), MDZ_THREADS, 0, st>>>(
                ns.nx, ns.nz, kind, kind, ns.X, ns.Z, g.dx, g.dz, g.ncx, g.ncz, ctx->bins.quads, ctx->bins.start,
                ctx->bins.sorted, ctx->m.x, ctx->m.z, ctx->m.phase, ctx->n_phases, dc, dp);
        MDZ_LAUNCHED(ctx);
        if (hc) MDZ_CUDA(ctx, cudaMemcpyAsync(hc, dc, sizeof(int) * nn, cudaMemcpyDeviceToHost, st));
        if (hp) MDZ_CUDA(ctx, cudaMemcpyAsync(hp, dp, sizeof(int) * (size_t)nn * ctx->n_phases, cudaMemcpyDeviceToHost, st));
        MDZ_CUDA(ctx, cudaStreamSynchronize(st));
    }
    return MDZ_OK;
}

// ---------------------------------------------------------------------------
// Grid -> marker.  Interp_Grid2P on a node set with lines X (n x) and Z (n z).
__device__ __forceinline__ bool air(signed char t) { return t == 30 || t == 31; }

__device__ double g2p_bilinear(double xk, double zk, const double *__restrict__ F, const double *__restrict__ X,
                               const double *__restrict__ Z, int Nx, int Nz, const signed char *__restrict__ tag,
                               double dx, double dz) {
    const double idx = 1.0 / dx, idz = 1.0 / dz;
    int jp = lower_line(xk, X[0], dx, idx);
    if (jp < 0) jp = 0;
    if (jp > Nx - 2) jp = Nx - 2;
    int ip = lower_line(zk, Z[0], dz, idz);
    if (ip < 0) ip = 0;
    if (ip > Nz - 2) ip = Nz - 2;
    double dxm = fabs(xk - X[jp]), dzm = fabs(zk - Z[ip]);
    int iSW = jp + ip * Nx, iSE = iSW + 1, iNW = jp + (ip + 1) * Nx, iNE = iNW + 1;
    double v = 0.0;
    const double wx = dxm * idx, wz = dzm * idz;
    v += (1.0 - wx) * (1.0 - wz) * (air(tag[iSW]) ? F[iNW] : F[iSW]);
    v += wx * (1.0 - wz) * (air(tag[iSE]) ? F[iNE] : F[iSE]);
    v += (1.0 - wx) * wz * (air(tag[iNW]) ? F[iSW] : F[iNW]);
    v += wx * wz * (air(tag[iNE]) ? F[iSE] : F[iNE]);
    return v;
}

__global__ void k_g2p_nodes(int n, const double *__restrict__ mx, const double *__restrict__ mz,
                            const int *__restrict__ mphase, const double *__restrict__ F, const double *__restrict__ X,
                            const double *__restrict__ Z, int Nx, int Nz, const signed char *__restrict__ tag,
                            double dx, double dz, double *__restrict__ out) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    if (mphase[k] == -1) { out[k] = 0.0; return; }
    out[k] = g2p_bilinear(mx[k], mz[k], F, X, Z, Nx, Nz, tag, dx, dz);
}

// Interp_Grid2P_centroids2, non-periodic: centroid field (ncx x ncz) in the
// ghosted frame xvz/zvx; outside ring rows/columns repeat the edge value.
__global__ void k_g2p_centroids_ext(int n, const double *__restrict__ mx, const double *__restrict__ mz,
                                    const int *__restrict__ mphase, const double *__restrict__ F,
                                    const double *__restrict__ xvz, const double *__restrict__ zvx, int ncx, int ncz,
                                    const signed char *__restrict__ tag, double dx, double dz,
                                    double *__restrict__ out) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    if (mphase[k] == -1) { out[k] = 0.0; return; }
    double xk = mx[k], zk = mz[k];
    const double idx = 1.0 / dx, idz = 1.0 / dz;
    int jp = lower_line(xk, xvz[0], dx, idx);
    int ip = lower_line(zk, zvx[0], dz, idz);
    int jw, je, is, in_;   // centroid columns west/east and rows south/north
    if (jp > 0 && jp < ncx) { jw = jp - 1; je = jp; }
    else if (jp <= 0) { jw = 0; je = 0; }
    else { jw = ncx - 1; je = ncx - 1; }
    if (ip > 0 && ip < ncz) { is = ip - 1; in_ = ip; }
    else if (ip <= 0) { is = 0; in_ = 0; }
    else { is = ncz - 1; in_ = ncz - 1; }
    int iSW = jw + is * ncx, iSE = je + is * ncx, iNW = jw + in_ * ncx, iNE = je + in_ * ncx;
    // clamp the line index used for the distances like the reference's ranges
    int jx = jp < 0 ? 0 : (jp > ncx ? ncx : jp);
    int iz = ip < 0 ? 0 : (ip > ncz ? ncz : ip);
    double dxm = xk - xvz[jx], dzm = zk - zvx[iz];
    double v = 0.0;
    const double wx = dxm * idx, wz = dzm * idz;
    v += (1.0 - wx) * (1.0 - wz) * (air(tag[iSW]) ? F[iNW] : F[iSW]);
    v += wx * (1.0 - wz) * (air(tag[iSE]) ? F[iNE] : F[iSE]);
    v += (1.0 - wx) * wz * (air(tag[iNW]) ? F[iSW] : F[iNW]);
    v += wx * wz * (air(tag[iNE]) ? F[iSE] : F[iNE]);
    out[k] = v;
}

extern "C" mdz_status mdz_Interp_Grid2P(mdz_ctx *ctx, const double *node_field, int node_set, double *marker_field) {
    if (!ctx) return MDZ_ERR_ARG;
    if (!node_field || !marker_field) return mdz_fail(ctx, MDZ_ERR_ARG, "Interp_Grid2P: null pointer");
    if (node_set < -2 || node_set > 1) return mdz_fail(ctx, MDZ_ERR_ARG, "Interp_Grid2P: bad node set");
    cudaStream_t st = ctx->stream;
    const mdz_dgrid &g = ctx->g;
    mdz_nodeset ns = mdz_get_nodeset(ctx, node_set);
    size_t nn = (size_t)ns.nx * ns.nz;
    int n = ctx->m.n;
    double *dF = (double *)mdz_stage(ctx, 0, sizeof(double) * nn);
    double *dO = (double *)mdz_stage(ctx, 1, sizeof(double) * (n ? n : 1));
    if (!dF || !dO) return mdz_fail(ctx, MDZ_ERR_CUDA, "Interp_Grid2P: staging allocation failed");
    MDZ_CUDA(ctx, cudaMemcpyAsync(dF, node_field, sizeof(double) * nn, cudaMemcpyHostToDevice, st));
    if (n > 0) {
        if (node_set == MDZ_NODES_CENTROIDS)
            k_g2p_centroids_ext<<<mdz_blocks(n), MDZ_THREADS, 0, st>>>(n, ctx->m.x, ctx->m.z, ctx->m.phase, dF, g.xvz,
                                                                       g.zvx, g.ncx, g.ncz, g.BCp, g.dx, g.dz, dO);
        else
            k_g2p_nodes<<<mdz_blocks(n), MDZ_THREADS, 0, st>>>(n, ctx->m.x, ctx->m.z, ctx->m.phase, dF, ns.X, ns.Z,
                                                               ns.nx, ns.nz, ns.tag, g.dx, g.dz, dO);
        MDZ_LAUNCHED(ctx);
        MDZ_CUDA(ctx, cudaMemcpyAsync(marker_field, dO, sizeof(double) * n, cudaMemcpyDeviceToHost, st));
    }
    MDZ_CUDA(ctx, cudaStreamSynchronize(st));
    return MDZ_OK;
}

// ---------------------------------------------------------------------------
// RK4 advection.  V2P without the conservative correction: Vx bilinear on
// (xg, zvx) and Vz on (xvz, zg), lower-left cell ceil(d/h) - 1 clamped to
// [0, N-2], tag-30 substitutions as in the reference.
//
// Both components need the position on the vertex lines and on the ghosted
// lines half a cell below: one fma gives both indices.
__device__ __forceinline__ void line_pair_indices(const line_pair &L, double x, int &i, int &ih) {
    if (!line_indices(x - L.X[0], L.ih, 0.0, L.off, i, ih)) {
        i = lower_line(x, L.X[0], L.h, L.ih);
        ih = lower_line(x, L.Xh[0], L.h, L.ih);
    }
    i = i < 0 ? 0 : (i > L.n - 2 ? L.n - 2 : i);
    ih = ih < 0 ? 0 : (ih > L.n - 1 ? L.n - 1 : ih);
}

__device__ __forceinline__ void v2p(double xk, double zk, const double *__restrict__ u, const double *__restrict__ v,
                                    const line_pair &LX, const line_pair &LZ, const signed char *__restrict__ tu,
                                    const signed char *__restrict__ tv, double &vxm, double &vzm) {
    int jg, jh, ig, ih;
    line_pair_indices(LX, xk, jg, jh);
    line_pair_indices(LZ, zk, ig, ih);
    // Vx: Nx x (Nz+1)
    {
        const int nx = LX.n;
        const double wx = fabs(xk - LX.X[jg]) * LX.ih, wz = fabs(zk - LZ.Xh[ih]) * LZ.ih;
        const int iSW = jg + ih * nx, iSE = iSW + 1, iNW = iSW + nx, iNE = iNW + 1;
        double VNW = u[iNW], VNE = u[iNE], VSW = u[iSW], VSE = u[iSE];
        if (tu[iSW] == 30) VSW = u[iNW];
        if (tu[iSE] == 30) VSE = u[iNE];
        if (tu[iNW] == 30) VNW = u[iSW];
        if (tu[iNE] == 30) VNE = u[iSE];
        if (tu[iNE] == 30 && tu[iSE] == 30) { VNE = VSW; VSE = VSW; }
        if (tu[iNW] == 30 && tu[iSW] == 30) { VNW = VSE; VSW = VSE; }
        const double v13 = VSW + wx * (VSE - VSW), v24 = VNW + wx * (VNE - VNW);
        vxm = v13 + wz * (v24 - v13);
    }
    // Vz: (Nx+1) x Nz
    {
        const int nx = LX.n + 1;
        const double wx = fabs(xk - LX.Xh[jh]) * LX.ih, wz = fabs(zk - LZ.X[ig]) * LZ.ih;
        const int iSW = jh + ig * nx, iSE = iSW + 1, iNW = iSW + nx, iNE = iNW + 1;
        double VSE = v[iSE], VSW = v[iSW], VNE = v[iNE], VNW = v[iNW];
        if (tv[iSW] == 30) VSW = v[iNE];
        if (tv[iSE] == 30) VSE = v[iNE];
        if (tv[iNW] == 30) VNW = v[iSW];
        if (tv[iNE] == 30) VNE = v[iSE];
        if (tv[iNE] == 30 && tv[iSE] == 30) { VNE = VSW; VSE = VSW; }
        if (tv[iNW] == 30 && tv[iSW] == 30) { VNW = VSE; VSW = VSE; }
        const double v12 = VSW + wz * (VNW - VSW), v34 = VSE + wz * (VNE - VSE);
        vzm = v12 + wx * (v34 - v12);
    }
}

// The box as keys whose integer order is that of the FP64 numbers: four FP64
// comparisons per stage would cost as much of that pipe as half a velocity.
struct box_keys { long long xmin, xmax, zmin, zmax; };

__host__ __device__ inline long long order_key(long long b) { return b ^ (long long)((unsigned long long)(b >> 63) >> 1); }

// x < xmin || x > xmax (false for a NaN)
__device__ __forceinline__ bool beyond(double x, long long kmin, long long kmax) {
    const long long b = __double_as_longlong(x), k = order_key(b);
    return (k < kmin || k > kmax) && (unsigned long long)(b & 0x7fffffffffffffffLL) <= 0x7ff0000000000000ULL;
}

// Bound by the FP64 pipe, 16 clocks per warp instruction: some 115 a marker.
// With ceil_quot for four indices per velocity, four comparisons per box test
// and weights in place of differences they were 265: 2.1 M markers 965 us,
// 535 with line_index, 472 with one fma for the two lines of a direction.
__global__ void k_rk4(int n, double *__restrict__ mx, double *__restrict__ mz, int *__restrict__ mphase,
                      double *__restrict__ mvx, double *__restrict__ mvz, const double *__restrict__ u,
                      const double *__restrict__ v, line_pair LX, line_pair LZ, const signed char *__restrict__ tu,
                      const signed char *__restrict__ tv, double dt, double dt_half, box_keys box) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    int ph = mphase[k];
    const double xA = mx[k], zA = mz[k];
    double x = xA, z = zA, Vx = 0, Vz = 0, sx = 0, sz = 0;   // stage velocity; A + 2 B + 2 C + D
#define OUT_CHECK() if (beyond(x, box.xmin, box.xmax) || beyond(z, box.zmin, box.zmax)) ph = -1;
    if (ph != -1) {
        v2p(x, z, u, v, LX, LZ, tu, tv, Vx, Vz);
        sx = Vx; sz = Vz;
        x = xA + dt_half * Vx; z = zA + dt_half * Vz;
    }
    OUT_CHECK();
    if (ph != -1) {
        v2p(x, z, u, v, LX, LZ, tu, tv, Vx, Vz);
        sx += 2.0 * Vx; sz += 2.0 * Vz;
        x = xA + dt_half * Vx; z = zA + dt_half * Vz;
    }
    OUT_CHECK();
    if (ph != -1) {
        v2p(x, z, u, v, LX, LZ, tu, tv, Vx, Vz);
        sx += 2.0 * Vx; sz += 2.0 * Vz;
        x = xA + dt * Vx; z = zA + dt * Vz;
    }
    OUT_CHECK();
    if (ph != -1) {
        v2p(x, z, u, v, LX, LZ, tu, tv, Vx, Vz);
        Vx = (1.0 / 6.0) * (sx + Vx); Vz = (1.0 / 6.0) * (sz + Vz);
        x = xA + dt * Vx; z = zA + dt * Vz;
        mvx[k] = Vx; mvz[k] = Vz;
    }
    OUT_CHECK();
#undef OUT_CHECK
    mx[k] = x; mz[k] = z; mphase[k] = ph;
}

mdz_status mdz_dev_rk4(mdz_ctx *ctx, const double *du, const double *dv, double dt, cudaStream_t st) {
    const mdz_dgrid &g = ctx->g;
    int n = ctx->m.n;
    if (n > 0) {
        auto key = [](double v, bool low) {   // a bound of zero holds -0 and +0
            long long b;
            memcpy(&b, &v, sizeof b);
            return v == 0.0 ? (low ? -1LL : 0LL) : order_key(b);
        };
        const box_keys box{key(g.xmin, true), key(g.xmax, false), key(g.zmin, true), key(g.zmax, false)};
        const mdz_grid_desc &hd = ctx->host_desc;
        k_rk4<<<mdz_blocks(n), MDZ_THREADS, 0, st>>>(n, ctx->m.x, ctx->m.z, ctx->m.phase, ctx->m.vx, ctx->m.vz, du, dv,
                                                     make_line_pair(g.xg, g.xvz, hd.xg[0], hd.xvz[0], g.dx, g.Nx),
                                                     make_line_pair(g.zg, g.zvx, hd.zg[0], hd.zvx[0], g.dz, g.Nz), g.BCu, g.BCv,
                                                     dt, 0.5 * dt, box);
        MDZ_LAUNCHED(ctx);
    }
    ctx->bins.valid = false;
    return MDZ_OK;
}

extern "C" mdz_status mdz_RogerGuntherII(mdz_ctx *ctx, const double *u, const double *v, double dt) {
    if (!ctx) return MDZ_ERR_ARG;
    if (!u || !v) return mdz_fail(ctx, MDZ_ERR_ARG, "RogerGuntherII: null velocity");
    cudaStream_t st = ctx->stream;
    const mdz_dgrid &g = ctx->g;
    size_t nu = (size_t)g.Nx * (g.Nz + 1), nv = (size_t)(g.Nx + 1) * g.Nz;
    double *du = (double *)mdz_stage(ctx, 0, sizeof(double) * nu);
    double *dv = (double *)mdz_stage(ctx, 1, sizeof(double) * nv);
    if (!du || !dv) return mdz_fail(ctx, MDZ_ERR_CUDA, "RogerGuntherII: staging allocation failed");
    MDZ_CUDA(ctx, cudaMemcpyAsync(du, u, sizeof(double) * nu, cudaMemcpyHostToDevice, st));
    MDZ_CUDA(ctx, cudaMemcpyAsync(dv, v, sizeof(double) * nv, cudaMemcpyHostToDevice, st));
    mdz_status s = mdz_dev_rk4(ctx, du, dv, dt, st);
    if (s != MDZ_OK) return s;
    MDZ_CUDA(ctx, cudaStreamSynchronize(st));
    return MDZ_OK;
}
