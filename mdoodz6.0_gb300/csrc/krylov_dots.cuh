// Inner products of the Krylov basis: (a_q, b) for a table of vectors in one
// launch, fixed-order sums.  Used by the sums of a Gram-Schmidt pass
// (k_gcr_dots in solver.cu) and by k_dots.
#pragma once
#include "mdz_internal.cuh"
#include "reduce.cuh"

template <typename T>
struct alignas(16) vec16 {
    static constexpr int N = 16 / sizeof(T);
    T v[N];
};

__device__ __forceinline__ double warp_sum_all(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// out[q] = (a_q, b) for the nq vectors of the pointer table (each of padded
// length n, contiguous u|v|p like b).  One thread keeps Q running sums and loads
// 16 bytes of each vector and of b at a time, so b is read once per Q vectors
// and the loads of all of them are in flight together.  FP32 vectors (Q = 8):
// products, sums and the warp reductions stay FP32 with only the warp sums
// entering FP64 (FP64 instructions issue at a small fraction of the FP32 rate
// on this part, so even a per-thread FP64 reduction tree dominated the
// kernel).  FP64 vectors (Q = 4) are bound by their FP64 multiply-adds.  Block
// row y handles vectors y Q .. y Q + Q - 1; its blocks write their partials to
// part[q * gridDim.x + blockIdx.x] and the last block of the row to finish
// adds them up in block order (reduce.cuh): deterministic.  cnt: one arrival
// counter per block row.
// 1025 x 513 in FP32, up to 8 / 16 / 24 vectors: 13.8 / 21.2 / 29.6 us, with
// 4-byte loads 18.9 / 32.7 / 51.7.
template <typename T>
constexpr int dots_q() { return sizeof(T) == 4 ? 8 : 4; }
// Block sums of Q FP64 values by 256 threads, valid in thread 0: 256 / Q threads
// per value fold the partial sums in shared memory and shuffle, 64 warp
// instructions on the FP64 pipe for Q = 4 (shuffles of every value in every warp
// took 160, and 20 more in the first).  Sums in a fixed order.
template <int Q>
__device__ __forceinline__ void dots_fold(const double (&p)[Q], double (&bs)[Q], double *sh) {
    static_assert(Q == 4, "64 threads per value");
    const int t = threadIdx.x;
#pragma unroll
    for (int j = 0; j < Q; j++) sh[j * 256 + t] = p[j];
    __syncthreads();
    const double *a = sh + (t >> 6) * 256 + (t & 63);
    const double s = warp_sum_all((a[0] + a[64]) + (a[128] + a[192]));
    if ((t & 31) == 0) sh[Q * 256 + (t >> 5)] = s;
    __syncthreads();
    if (t == 0)
#pragma unroll
        for (int j = 0; j < Q; j++) bs[j] = sh[Q * 256 + 2 * j] + sh[Q * 256 + 2 * j + 1];
}
template <typename T, int MDOT_Q>
constexpr int dots_shared() { return sizeof(T) == 8 ? MDOT_Q * 256 + 8 : 32 * MDOT_Q; }
// p += the products of one load.  In FP32 the four are added up in pairs first, so
// that a thread's chain of FP32 additions has a link per load and not per
// element: 13 loads at 1025 x 513 and 34 vectors are a chain of 16 (50 one by
// one; the two products more a load cost nothing beside its traffic).
__device__ __forceinline__ void dots_add(float &p, const vec16<float> &a, const vec16<float> &b) {
    p += (a.v[0] * b.v[0] + a.v[1] * b.v[1]) + (a.v[2] * b.v[2] + a.v[3] * b.v[3]);
}
__device__ __forceinline__ void dots_add(double &p, const vec16<double> &a, const vec16<double> &b) {
#pragma unroll
    for (int e = 0; e < 2; e++) p += a.v[e] * b.v[e];
}
// (b: the vector as a function of the position; self: the place among the Q of
// (b, b), whose ap is not read, or -1)
template <typename T, int MDOT_Q, typename VEC>
__device__ __forceinline__ void dots_block(int nq, size_t n, const T *const *ap, const VEC &b, int self,
                                           double *part, double (&bs)[MDOT_Q], double *sh) {
    typedef vec16<T> V;
    T p[MDOT_Q];
#pragma unroll
    for (int j = 0; j < MDOT_Q; j++) p[j] = T(0);
    const size_t stride = (size_t)gridDim.x * blockDim.x * V::N;
    for (size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * V::N; i < n; i += stride) {
        const V bi = b(i);
        V a[MDOT_Q];
#pragma unroll
        for (int j = 0; j < MDOT_Q; j++) {
            if (j == self) a[j] = bi;
            else if (ap[j]) a[j] = *reinterpret_cast<const V *>(ap[j] + i);
        }
#pragma unroll
        for (int j = 0; j < MDOT_Q; j++)
            if (ap[j]) dots_add(p[j], a[j], bi);
    }
    if constexpr (sizeof(T) == 8) dots_fold<MDOT_Q>(p, bs, sh);
    else mdz_block_sum<MDOT_Q, T>(p, bs, sh);
    const int q0 = blockIdx.y * MDOT_Q;
    if (threadIdx.x == 0) {
#pragma unroll
        for (int j = 0; j < MDOT_Q; j++)
            if (q0 + j < nq) part[(size_t)(q0 + j) * gridDim.x + blockIdx.x] = bs[j];
    }
}

template <typename T, int MDOT_Q>
__global__ void __launch_bounds__(256) k_dots(int nq, size_t n, const T *const *__restrict__ a,
                                              const T *__restrict__ b, double *part, unsigned int *cnt,
                                              double *out) {
    __shared__ double sh[dots_shared<T, MDOT_Q>()];
    const int q0 = blockIdx.y * MDOT_Q;
    const T *ap[MDOT_Q];
#pragma unroll
    for (int j = 0; j < MDOT_Q; j++) ap[j] = q0 + j < nq ? a[q0 + j] : nullptr;
    double bs[MDOT_Q];
    dots_block<T, MDOT_Q>(nq, n, ap, [&](size_t i) { return *reinterpret_cast<const vec16<T> *>(b + i); }, -1, part, bs, sh);
    if (!mdz_arrive_last(cnt + blockIdx.y, gridDim.x)) return;
    const int nrow = nq - q0 < MDOT_Q ? nq - q0 : MDOT_Q;
    mdz_sum_partials(part + (size_t)q0 * gridDim.x, gridDim.x, nrow, out + q0);
}

// grid of a dots launch over nq vectors: block rows of Q vectors, about four
// blocks per SM in all, each thread at least one 16-byte load per vector
template <typename T>
static dim3 dots_grid(size_t n, int nq) {
    constexpr int Q = dots_q<T>();
    const int rows = (nq + Q - 1) / Q;
    int bx = mdz_blocks((long long)n, 256 * vec16<T>::N);
    const int cap = (152 * 4 + rows - 1) / rows;
    if (bx > cap) bx = cap;
    return dim3(bx, rows);
}
