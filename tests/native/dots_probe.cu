// k_dots on its own, for tests/test_dots_chain_gpu.py: out[q] = (a_q, b) of nq
// FP32 vectors of n elements (n a multiple of 32), with the launch's own grid.
#include <vector>
#include "krylov_dots.cuh"

extern "C" int probe_dots(int nq, long long n, const float *a, const float *b, double *out) {
    float *d = nullptr;
    const float **tab = nullptr;
    double *part = nullptr;
    unsigned int *cnt = nullptr;
    const dim3 gr = dots_grid<float>((size_t)n, nq);
    cudaMalloc((void **)&d, sizeof(float) * n * (nq + 1));
    cudaMalloc((void **)&tab, sizeof(float *) * nq);
    cudaMalloc((void **)&part, sizeof(double) * (gr.x * gr.y * dots_q<float>() + nq));
    cudaMalloc((void **)&cnt, sizeof(int) * gr.y);
    std::vector<const float *> t(nq);
    for (int q = 0; q < nq; q++) t[q] = d + (size_t)q * n;
    cudaMemcpy(d, a, sizeof(float) * n * nq, cudaMemcpyHostToDevice);
    cudaMemcpy(d + (size_t)nq * n, b, sizeof(float) * n, cudaMemcpyHostToDevice);
    cudaMemcpy(tab, t.data(), sizeof(float *) * nq, cudaMemcpyHostToDevice);
    cudaMemset(cnt, 0, sizeof(int) * gr.y);
    double *res = part + (size_t)gr.x * gr.y * dots_q<float>();
    if (cudaGetLastError() == cudaSuccess)
        k_dots<float, dots_q<float>()><<<gr, 256>>>(nq, (size_t)n, tab, d + (size_t)nq * n, part, cnt, res);
    cudaMemcpy(out, res, sizeof(double) * nq, cudaMemcpyDeviceToHost);
    const int e = (int)cudaDeviceSynchronize();
    cudaFree(d); cudaFree(tab); cudaFree(part); cudaFree(cnt);
    return e;
}
