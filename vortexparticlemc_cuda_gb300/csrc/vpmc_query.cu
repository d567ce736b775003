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

// Field values at scattered points, one warp a point, lanes over the particles of
// the walk (which is trimmed to the point itself: the columns and sub-rows within
// reach of it).  Lanes over the points of a bin (k_eval) leave most lanes idle when
// a bin holds a few points; here a point costs about 0.6 instructions a visited
// particle against 0.2 for a full bin of 128 points, and a point has a price of its own
// (0.4 ns) that binned ones have not.  Gathered are up to kGatherPoints points a
// half-support cell of up to kGatherSome; up to kGatherMost with at most kGatherPairs
// particles in reach of them in all (so few points leave the device idle when they are
// binned); and any number where the cells hold kGatherSparse points or fewer (us a call
// gathered / binned: 50,000 points in 200^2 particles, h_w 16 spacings: 167 / 316; 200,000 in
// 600,000, h_w 0.02, 20 a cell: 369 / 390, 400,000, 40 a cell: 596 / 401; 1,000,000 in
// 300,000, h_w 0.01, 25 a cell: 608 / 286; h_w 0.002, 1 a cell: 502 / 562; 3,000,000,
// 3 a cell: 1,213 / 669).  Needs no binning of the points.  20,011 points in 262,144
// particles, h_w = 16 spacings: 224 us binned (half-support cells), 36 us gathered; the
// whole call 401 -> 143 us.
constexpr double kGatherPoints = 40.0;
constexpr long kGatherSome = 3L << 16;
constexpr long kGatherMost = 1L << 17;
constexpr double kGatherPairs = double(1L << 27);
constexpr double kGatherSparse = 1.0;
// Binned points take cells a quarter as full as a simulation's samples do (37 points):
// 476,719 points in 422^2 particles, h_w 16 spacings: 557 -> 424 us, 700,000 in 300^2,
// h_w 8: 445 -> 338 us.
constexpr double kBinShare = 4.0;
constexpr double kCrowdedCell = 64.0;     // points a half-support cell
constexpr double kCrowdedPairs = 7000.0;  // and particles in reach of each
constexpr int kGatherRows = 4;   // sub-rows a cell
// Sub-rows a cell for binned points: 16, halved until the grid has at most 2^22, and no more
// than 8 a particle or 1 for 16 points (each is a search and 4 bytes).  h_w = 0.001 of the
// period, 4 M cells: deformed queries of 100 points in 100 particles 360 us with 16, 245
// with 1 (271 once), FP64 ones 394 and 234; h_w = 0.1, 300,000 points in 10,000 particles:
// 489 with 16, 583 with 1, 1,000,000 in 100: 511 and 568.
constexpr int kQueryRows = 16;
constexpr double kMostSubRows = double(1L << 22);

// For k cells a h_w at the reach h_w cover.
int query_rows(long N, long M, float hw, float cover, float Lx, float Ly, int k) {
    const double reach = double(hw) * cover, cells = (double(k) * Lx / reach) * (double(k) * Ly / reach);
    const double most = std::min(kMostSubRows, std::max(8.0 * double(N), double(M) / 16.0));
    int rows = kQueryRows;
    while (rows > 1 && cells * rows > most) rows /= 2;
    return rows;
}

__global__ void k_gather_records(const uint32_t* __restrict__ perm, const uint32_t* __restrict__ start, long n, long nsub,
                                 const float2* __restrict__ pos, const float* __restrict__ omega,
                                 const GridInst* __restrict__ inst, int set_mode, double two_sigma,
                                 float4* __restrict__ rec) {
    const long nv = min(long(start[nsub]), n);
    const GridInst& G = inst[0];
    for (long p = long(blockIdx.x) * blockDim.x + threadIdx.x; p < nv; p += long(gridDim.x) * blockDim.x) {
        const uint32_t i = perm[p];
        float2 q = pos[i];
        if (G.periodic) {
            q.x = q.x - floorf(q.x / G.Lx) * G.Lx;
            q.y = q.y - floorf(q.y / G.Ly) * G.Ly;
        }
        const float w = omega[i];
        rec[p] = make_float4(q.x, q.y, float(double(set_mode == SET_ONE_SIGNED ? w : fabsf(w)) * two_sigma), 0.f);
    }
}

template <bool EXC>
__global__ void __launch_bounds__(256) k_gather_points(const GridInst* __restrict__ inst,
                                                       const uint32_t* __restrict__ start, int rows,
                                                       const float4* __restrict__ rec, const float2* __restrict__ pts,
                                                       long M, float* __restrict__ out) {
    const GridInst& G = inst[0];
    const int lane = threadIdx.x & 31;
    const long warp = (long(blockIdx.x) * blockDim.x + threadIdx.x) >> 5, nwarps = (long(gridDim.x) * blockDim.x) >> 5;
    const int gyR = G.gy * rows;
    const float sx = 1.f / G.inv_sx, inv_srow = G.inv_sy * float(rows), rm = G.reach * 1.001f;
    const float kap = G.B;   // -3 / h^2, see packed_run of the evaluation kernel
    for (long m = warp; m < M; m += nwarps) {
        float2 p = pts[m];
        bool ok = p.x == p.x && p.y == p.y;
        if (ok && G.periodic) {
            p.x = p.x - floorf(p.x / G.Lx) * G.Lx;
            p.y = p.y - floorf(p.y / G.Ly) * G.Ly;
        } else if (ok) {
            ok = !(p.x < 0.f || p.x > G.Lx || p.y < 0.f || p.y > G.Ly);
        }
        // lane c: column c - k of the walk, its sub-rows within reach of the point
        uint32_t beg[2] = {0u, 0u}, end[2] = {0u, 0u};
        int sxi = 0, syi[2] = {0, 0};
        if (ok && lane <= 2 * G.k) {
            const int cx = min(max(floor_int(p.x * G.inv_sx), 0), G.gx - 1);
            int gxx = cx + lane - G.k;
            const float x0 = float(gxx) * sx, dx = fmaxf(0.f, fmaxf(x0 - p.x, p.x - (x0 + sx)));
            bool col = dx < rm;
            if (G.periodic) {
                if (gxx < 0) { gxx += G.gx; sxi = -1; }
                else if (gxx >= G.gx) { gxx -= G.gx; sxi = 1; }
            } else if (gxx < 0 || gxx >= G.gx) {
                col = false;
            }
            if (col) {
                const float dy = sqrtf(fmaf(rm, rm, -dx * dx));
                int lo = floor_int(fmaf(p.y - dy, inv_srow, -0.01f)), hi = floor_int(fmaf(p.y + dy, inv_srow, 0.01f));
                int r0[2] = {1, 1}, r1[2] = {0, 0};
                if (!G.periodic) {
                    r0[0] = max(lo, 0);
                    r1[0] = min(hi, gyR - 1);
                } else if (lo < 0) {
                    r0[0] = 0; r1[0] = hi;
                    r0[1] = max(lo + gyR, hi + 1); r1[1] = gyR - 1; syi[1] = -1;
                } else if (hi >= gyR) {
                    r0[0] = lo; r1[0] = gyR - 1;
                    r0[1] = 0; r1[1] = min(hi - gyR, lo - 1); syi[1] = 1;
                } else {
                    r0[0] = lo; r1[0] = hi;
                }
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (r0[h] <= r1[h]) {
                        const uint32_t b0 = uint32_t(gxx * gyR + r0[h]);
                        beg[h] = start[b0];
                        end[h] = start[b0 + uint32_t(r1[h] - r0[h]) + 1u];
                    }
            }
        }
        float acc = 0.f;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            for (unsigned todo = __ballot_sync(0xffffffffu, end[h] > beg[h]); todo; todo &= todo - 1u) {
                const int c = __ffs(int(todo)) - 1;
                const uint32_t b = __shfl_sync(0xffffffffu, beg[h], c), e = __shfl_sync(0xffffffffu, end[h], c);
                const int ix = __shfl_sync(0xffffffffu, sxi, c), iy = __shfl_sync(0xffffffffu, syi[h], c);
                // image shift on whichever of particle and point makes it exact
                const float cx = ix < 0 ? -G.Lx : 0.f, cy = iy < 0 ? -G.Ly : 0.f;
                const float qx = ix > 0 ? p.x - G.Lx : p.x, qy = iy > 0 ? p.y - G.Ly : p.y;
#pragma unroll 4
                for (uint32_t i = b + uint32_t(lane); i < e; i += 32u) {
                    const float4 r = rec[i];
                    const float dx = (r.x + cx) - qx, dy = (r.y + cy) - qy;
                    const float r2 = fmaf(dx, dx, dy * dy), s2 = kap * r2;
                    const float t = __saturatef(fmaf(-kInvSqrt3, sqrt_approx(-s2), 1.f));
                    float v = fminf(fmaf(s2, t, 0.5f), t * t * t);
                    if (EXC && r2 < 1e-12f) v = 0.f;
                    acc = fmaf(r.z, v, acc);
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) out[m] = acc;
    }
}

__global__ void k_axpby(const double* __restrict__ a, const double* __restrict__ b, long n, double sa, double sb,
                        double* __restrict__ out) {
    for (long i = long(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += long(gridDim.x) * blockDim.x)
        out[i] = sa * a[i] + sb * b[i];
}

// The gather path of vpmc_query_vorticity: grid, compact records, one launch over the points.
int query_gather(vpmc_context* ctx, long N, const float2* pos, const float* omega, long M, const float2* pts, int set_mode,
                 bool exclude, float hw, float Lx, float Ly, int periodic, float* out) {
    cudaStream_t st = ctx->stream;
    // columns of about 48 particles or more keep the lanes busy
    const double density = double(N) / (double(Lx) * Ly);
    const int k = int(std::min(3.0, std::max(1.0, 2.0 * double(hw) * hw * density / 48.0)));
    InstDesc d{Lx, Ly, hw, periodic, 0, int(N)};
    d.k = double(k) * Lx / hw * k * Ly / hw <= double(1L << 22) ? k : 1;
    GridInst plan;
    const long nb = grid_plan(&d, 1, 0, 1, &plan);
    if (nb < 0) return int(-nb);
    GridBufs g;
    float4* rec = nullptr;
    auto carve = [&](Carver& c) {
        carve_grid(c, N, nb, 1, &g, false, kGatherRows, false);
        rec = c.take<float4>(size_t(N));
    };
    Carver dry;
    carve(dry);
    char* base = nullptr;
    VPMC_TRY(scratch(ctx, SLOT_QUERY, dry.off, &base));
    Carver c{base, 0};
    carve(c);
    VPMC_CUDA(cudaMemcpyAsync(g.inst, &plan, sizeof(GridInst), cudaMemcpyHostToDevice, st));
    VPMC_TRY(grid_sort(ctx, g, pos, omega, set_mode));
    const double two_sigma = 80.0 / (7.0 * kPiD * double(hw) * hw);
    VPMC_LAUNCH(k_gather_records, work_blocks(N), 256, 0, st, g.perm, g.start, N, nb * kGatherRows, pos, omega, g.inst,
                set_mode, two_sigma, rec);
    const int grid = int(std::min<long>((M + 7) / 8, 8L * ctx->sm_count));
    if (exclude) VPMC_LAUNCH(k_gather_points<true>, grid, 256, 0, st, g.inst, g.start, kGatherRows, rec, pts, M, out);
    else VPMC_LAUNCH(k_gather_points<false>, grid, 256, 0, st, g.inst, g.start, kGatherRows, rec, pts, M, out);
    return VPMC_OK;
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
    const int set_mode = sign > 0 ? SET_POS_ONLY
                                   : (sign < 0 ? SET_NEG_ONLY : (use_signed ? SET_ONE_SIGNED : SET_ONE_ABS));
    // (the gathered form has no staging wait to give up: a limit of 0 polls keeps the
    // binned one, whose first wait then expires)
    const double reach = 3.14159265 * double(N) * h_w * h_w / (double(Lx) * Ly);   // particles within h_w
    const double per_cell = double(M) / ((2.0 * Lx / h_w) * (2.0 * Ly / h_w));
    const bool few = per_cell <= kGatherSparse || (M <= kGatherSome && per_cell <= kGatherPoints) ||
                     (M <= kGatherMost && double(M) * reach <= kGatherPairs);
    if (!F && ctx->wait_limit > 0 && few) {
        VPMC_TRY(query_gather(ctx, N, reinterpret_cast<const float2*>(pos), omega, M, reinterpret_cast<const float2*>(pts),
                              set_mode, exclude_center != 0, h_w, Lx, Ly, periodic, out));
        if (sign < 0 && use_signed) VPMC_LAUNCH(k_scale_f32, work_blocks(M), 256, 0, st, out, long(M), -1.0f);
        return vpmc_context_sync(ctx);
    }
    Work w;
    // smaller cells and sub-rows trim the walk, as in a simulation's passes
    // one cell a h_w only while its bins are not crowded (the points of a bin are counted and
    // placed one after the other: 1,000,000 points, 100 particles, h_w 0.05: 470 us with 400
    // bins, 227 with 1,600; 1,000,000, 10,000, h_w 0.01, 100 a bin: 221 and 259) and their
    // pairs are few (200,000 points, 600,000 particles, h_w 0.02: 506 and 390)
    int k = F ? default_k() : sample_k(N, kBinShare * M, Lx, Ly, h_w);
    if (k == 1 && (per_cell > kCrowdedCell || per_cell * reach > kCrowdedPairs)) k = default_k();
    VPMC_TRY(setup_work(ctx, SLOT_QUERY, N, h_w, Lx, Ly, periodic, M, 0, &w, k, cover, F != nullptr,
                        query_rows(N, M, h_w, cover, Lx, Ly, k)));
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
    VPMC_TRY(setup_work(ctx, SLOT_QUERY, N, h_w, Lx, Ly, periodic, M, 0, &w, 0, 1.f, false,
                        query_rows(N, M, h_w, 1.f, Lx, Ly, default_k())));
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
