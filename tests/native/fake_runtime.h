// Stand-ins for CUDA runtime calls, put in front of a library source by the
// compiler's -include: what a device that cannot place a launch answers.
#pragma once
#include <cuda_runtime.h>

#ifdef FAKE_REFUSED_LAUNCHES
#define cudaLaunchCooperativeKernel(...) cudaErrorCooperativeLaunchTooLarge
template <typename K>
static cudaError_t no_clusters(int *n, K, const cudaLaunchConfig_t *) {
    *n = 0;
    return cudaSuccess;
}
template <typename K, typename... A>
static cudaError_t launch_without_clusters(const cudaLaunchConfig_t *cfg, K k, A... a) {
    for (unsigned i = 0; i < cfg->numAttrs; i++)
        if (cfg->attrs[i].id == cudaLaunchAttributeClusterDimension) return cudaErrorLaunchOutOfResources;
    return cudaLaunchKernelEx(cfg, k, a...);
}
#define cudaOccupancyMaxActiveClusters(...) no_clusters(__VA_ARGS__)
#define cudaLaunchKernelEx(...) launch_without_clusters(__VA_ARGS__)
#endif

#ifdef FAKE_RECORD_LIMITS
// every limit of dynamic shared memory that a kernel of this source was given
extern "C" {
inline int probe_limits_n = 0, probe_limits[64];
__attribute__((used)) inline int *probe_limits_get(int *n) { *n = probe_limits_n; return probe_limits; }
}
template <typename F>
static cudaError_t probe_set_attribute(F f, cudaFuncAttribute a, int v) {
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize && probe_limits_n < 64) probe_limits[probe_limits_n++] = v;
    return cudaFuncSetAttribute(f, a, v);
}
#define cudaFuncSetAttribute(f, a, v) probe_set_attribute(f, a, v)
#endif
