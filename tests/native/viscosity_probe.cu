// The local rheology of a context's nodes in either precision, for
// tests/test_rheology_fp32_gpu.py (the time step chooses the precision itself).
#include "mdz_internal.cuh"

extern "C" int probe_viscosity(mdz_ctx *ctx, const mdz_materials *m, const mdz_rheo_params *prm, mdz_fields *h, int fp32) {
    static const char *const out[] = {"eta_n", "eta_s", "sxxd", "szzd", "sxz", "eII_pwl", "eII_lin", "eII_pl", "exx_diss"};
    cudaStream_t st = ctx->stream;
    mdz_status s;
    if ((s = mdz_ensure_fields(ctx)) != MDZ_OK || (s = mdz_upload_fields(ctx, h, st)) != MDZ_OK ||
        (s = mdz_dev_viscosity(ctx, m, prm, ctx->d, ctx->d_counters, st, false, fp32 != 0)) != MDZ_OK ||
        (s = mdz_download_fields(ctx, h, out, 9, st)) != MDZ_OK)
        return s;
    return cudaStreamSynchronize(st) == cudaSuccess ? MDZ_OK : MDZ_ERR_CUDA;
}
