// vpmc_query.cu -- vorticity queries at arbitrary points on the evaluation grid
// of vpmc_grid.cu.
#include <algorithm>
#include <cmath>

#include "vpmc_work.cuh"

namespace vpmc {
namespace {

__global__ void k_scale_f32(float* __restrict__ a, long n, float s) {
    for (long i = long(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += long(gridDim.x) * blockDim.x) a[i] *= s;
}

__global__ void k_axpby(const double* __restrict__ a, const double* __restrict__ b, long n, double sa, double sb,
                        double* __restrict__ out) {
    for (long i = long(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += long(gridDim.x) * blockDim.x)
        out[i] = sa * a[i] + sb * b[i];
}

}  // namespace
}  // namespace vpmc

using namespace vpmc;

extern "C" {

int vpmc_query_vorticity(vpmc_context* ctx, int N, const float* pos, const float* omega, const float* F, int M,
                         const float* pts, int sign, int use_signed, int exclude_center, float h_w, float Lx,
                         float Ly, int periodic, float* out) {
    if (!ctx || N < 0 || M < 0 || !(h_w > 0.f) || !(Lx > 0.f) || !(Ly > 0.f)) return VPMC_ERR_INVALID;
    if ((N > 0 && (!pos || !omega)) || (M > 0 && (!pts || !out))) return VPMC_ERR_INVALID;
    VPMC_CUDA(cudaSetDevice(ctx->device));
    if (M == 0) return VPMC_OK;
    cudaStream_t st = ctx->stream;
    VPMC_CUDA(cudaMemsetAsync(out, 0, sizeof(float) * size_t(M), st));
    if (N == 0) return vpmc_context_sync(ctx);
    // deformed kernels: the walk must reach sigma_max(F) h_w (at most 2 h_w,
    // the reach of the reference's 3x3 walk of 2 h_w cells)
    float cover = 1.f;
    if (F) {
        char* sb = nullptr;
        VPMC_TRY(scratch(ctx, SLOT_MISC, 64, &sb));
        float sig = 1.f;
        VPMC_TRY(grid_max_sigma(ctx, reinterpret_cast<const float4*>(F), N, reinterpret_cast<unsigned*>(sb), &sig));
        if (!(sig <= 3.0e38f)) return VPMC_ERR_INVALID;   // non-finite F or det F <= 0
        cover = sig > 1.f ? std::min(2.f, std::ceil(sig * 16.f) / 16.f) : 1.f;
    }
    Work w;
    VPMC_TRY(setup_work(ctx, SLOT_QUERY, N, h_w, Lx, Ly, periodic, M, 0, &w, 0, cover, F != nullptr));
    const int set_mode = sign > 0 ? SET_POS_ONLY
                                   : (sign < 0 ? SET_NEG_ONLY : (use_signed ? SET_ONE_SIGNED : SET_ONE_ABS));
    VPMC_TRY(grid_build(ctx, w.g, reinterpret_cast<const float2*>(pos), omega, set_mode,
                        reinterpret_cast<const float4*>(F)));
    VPMC_TRY(bin_points(ctx, w.g, w.q, reinterpret_cast<const float2*>(pts), M, 0, 0));
    VPMC_TRY(make_items(ctx, w.g, w.q.qstart, w.it, query_chunk(4), M));
    EvalLaunch L;
    if (F) L.mode = exclude_center ? EVAL_FIELD_F_EXC : EVAL_FIELD_F;
    else L.mode = exclude_center ? EVAL_FIELD_EXC : EVAL_FIELD;
    L.out_f32 = out;
    VPMC_TRY(launch_eval(ctx, w.g, w.q.qrec, w.it, L));
    if (sign < 0 && use_signed) VPMC_LAUNCH(k_scale_f32, work_blocks(M), 256, 0, st, out, long(M), -1.0f);
    return vpmc_context_sync(ctx);
}

int vpmc_query_vorticity_f64(vpmc_context* ctx, int N, const float* pos, const float* omega, int M, const float* pts,
                             int sign, int use_signed, float h_w, float Lx, float Ly, int periodic, double* out) {
    if (!ctx || N < 0 || M < 0 || !(h_w > 0.f) || !(Lx > 0.f) || !(Ly > 0.f)) return VPMC_ERR_INVALID;
    if ((N > 0 && (!pos || !omega)) || (M > 0 && (!pts || !out))) return VPMC_ERR_INVALID;
    VPMC_CUDA(cudaSetDevice(ctx->device));
    if (M == 0) return VPMC_OK;
    cudaStream_t st = ctx->stream;
    VPMC_CUDA(cudaMemsetAsync(out, 0, sizeof(double) * size_t(M), st));
    if (N == 0) return vpmc_context_sync(ctx);
    Work w;
    VPMC_TRY(setup_work(ctx, SLOT_QUERY, N, h_w, Lx, Ly, periodic, M, 0, &w));
    const int set_mode = sign > 0 ? SET_POS_ONLY
                                   : (sign < 0 ? SET_NEG_ONLY : (use_signed ? SET_ONE_SIGNED : SET_ONE_ABS));
    VPMC_TRY(grid_build(ctx, w.g, reinterpret_cast<const float2*>(pos), omega, set_mode));
    VPMC_TRY(bin_points(ctx, w.g, w.q, reinterpret_cast<const float2*>(pts), M, 0, 0));
    VPMC_TRY(make_items(ctx, w.g, w.q.qstart, w.it, query_chunk(4), M));
    EvalLaunch L;
    L.mode = EVAL_FIELD64;
    L.out_f64 = out;
    VPMC_TRY(launch_eval(ctx, w.g, w.q.qrec, w.it, L));
    if (sign < 0 && use_signed)
        VPMC_LAUNCH(k_axpby, work_blocks(M), 256, 0, st, out, out, long(M), -1.0, 0.0, out);
    return vpmc_context_sync(ctx);
}

}  // extern "C"
