// vpmc_adjoint.cu -- the adjoint of the plain MIS step (no counterpart in
// the reference): checkpointed forward record, segment recompute, and per
// step the value/gradient field sums at the samples, the per-sample
// derivatives of the MIS term and the transposed field sum at the particles,
// each term in the forward's precision.  FP64 path: every sum in FP64.  FP32
// path: the sums over candidate runs and over a warp's samples as three floats
// (more digits than FP64), a sample's value and gradient rounded once to FP32
// (its terms read them so), what goes across warps and work items in FP64.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "vpmc_sim.cuh"
#include "vpmc_wide.cuh"

namespace vpmc {
namespace {

using namespace sim;

// ------------------------------------------------------------------ adjoint
// The adjoint of one plain MIS step X' = X + dt U(X, omega) with the step's
// Philox samples held fixed (common random numbers; the discrete CDF index
// and image-tile choices are constants of the pathwise derivative).  With
// lambda' = dL/dX' and v_t = dt lambda'_t (+-1/Q per sign), each MIS term
// T(x_t, y, f(y), Omega) contributes c = v_t . T and
//   dL/dx_t   += dc/dx                       (and dc/dy for disk samples, y = x_t + offset)
//   dL/dx_I   += dc/dy                       (branch-1 samples, y = x_I + shift + F r)
//   dc/dy      = -dc/dx|_f + dc/df grad f(y)
//   dL/domega_J, dL/dx_J through f(y) = sum_J |omega_J| W(|y - x_J|):
//              sgn(omega_J) G(x_J) and |omega_J| grad G(x_J), G(q) = sum_s dc_s/df W(|q - y_s|)
//              (the transposed field sum, evaluated with queries and candidates swapped)
//   dL/domega_J through Omega: sgn(omega_J) (9 if periodic) sum_s dc_s/dOmega.

// d(v . T)/d{x, f, Omega} of one MIS term (mis_term64's arithmetic), in R
// arithmetic: FP64 on the FP64 path, FP32 on the FP32 path (each term is then
// as precise as the forward's FP32 term; the caller sums in FP64 or three floats).
// The factor 1 - (w1 f / cum) / D of df/f is written as the disk term's share
// w2 p2 / D, which equals it and has no cancellation when branch 1 dominates.
// With E = w1 f r + w2a cum = D cum r the term needs the reciprocals of E and r^2
// alone (w2a: w2 alpha, icum: 1 / cum) instead of eight quotients.
template <typename R_>
__device__ __forceinline__ void mis_term_adj(int law, float2 xf, float2 yf, R_ f, R_ w1, R_ w2a, R_ cum, R_ icum,
                                             R_ R, const InstMC& I, R_ vx, R_ vy, R_& gxx, R_& gxy, R_& df, R_& dc,
                                             R_& cval) {
    gxx = gxy = df = dc = cval = R_(0);
    if (!(f > R_(0))) return;
    const R_ rx = R_(xf.x) - R_(yf.x), ry = R_(xf.y) - R_(yf.y);
    const R_ P = vy * rx - vx * ry;   // v . perp(r)
    const R_ i2pi = R_(0.5 / kPiD);
    if (law == VPMC_LAW_REFERENCE) {
        R_ wx = rx, wy = ry;
        if (I.periodic) {
            wx = rx - round(rx / R_(I.Lx)) * R_(I.Lx);
            wy = ry - round(ry / R_(I.Ly)) * R_(I.Ly);
        }
        const R_ wn = sqrt(wx * wx + wy * wy);
        const R_ rn = fmax(wn, R_(1e-6)), irn = R_(1) / rn;
        const R_ inv = R_(1) / (rx * rx + ry * ry + R_(1e-8));
        const R_ K = inv * i2pi;
        const R_ own = w1 * f * rn, disk = w2a * cum, iE = R_(1) / (own + disk);
        const R_ share = disk * iE, iD = cum * rn * iE;   // the disk term's share of the denominator, its reciprocal
        const R_ sc = f * iD;
        const R_ g = wn > R_(1e-6) ? sc * share * irn * irn : R_(0);   // d sc / d rn, over rn
        cval = sc * K * P;
        gxx = sc * K * vy - R_(2) * rx * inv * K * sc * P + K * P * g * wx;
        gxy = -sc * K * vx - R_(2) * ry * inv * K * sc * P + K * P * g * wy;
        df = K * P * share * iD;
        dc = K * P * sc * (own * iE * icum);
        return;
    }
    const R_ r2 = rx * rx + ry * ry;
    if (!(r2 > R_(0))) return;
    const R_ rn = sqrt(r2), ir2 = R_(1) / r2;
    const R_ own = w1 * f * rn, disk = rn < R ? w2a * cum : R_(0), iE = R_(1) / (own + disk);
    const R_ share = disk * iE, A = cum * rn * iE * (ir2 * i2pi);
    const R_ sc = f * A;
    const R_ ex = (R_(2) - share) * ir2;   // -(d sc / d r) / (sc r)
    cval = sc * P;
    gxx = sc * vy - P * sc * ex * rx;
    gxy = -sc * vx - P * sc * ex * ry;
    df = P * share * A;
    dc = P * sc * (own * iE * icum);
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

struct AdjArgs {
    const InstMC* mc;
    int n_inst;
    const float2* pos;
    const float2* ys;
    const double* fg;       // 3 per sample: f, df/dx, df/dy (FP64 path)
    const float* fg32;      // the same (FP32 path)
    const int* src;
    const double* cum64;    // 2 per instance (x9 when periodic)
    long t0, nt;
    int N1, N2;
    const double* lam_next;
    double* lam;
    double* as;             // per sample: dc/df
    double* dcum;           // 2 per instance
    double* gsc;            // score-function term: per particle, sum of c over the samples that drew it
    double* csum;           // 2 per instance: sum of c over branch-1 samples
};

// A lane's sum: FP64, or (FP32 path) three floats, which add FP32 terms with more
// digits than FP64 and without its 64-fold price.
template <bool F32>
struct AdjSum {
    double d = 0.0;
    __device__ __forceinline__ void add(double x) { d += x; }
    __device__ __forceinline__ double value() const { return d; }
};
template <>
struct AdjSum<true> {
    float s[3] = {0.f, 0.f, 0.f};
    __device__ __forceinline__ void add(float x) { wide::add_float(s, x); }
    __device__ __forceinline__ double value() const { return (double(s[0]) + double(s[1])) + double(s[2]); }
};

// One warp per target at a time: the MIS-term derivatives of all its samples, each in
// FP32 (F32: the FP32 path) or FP64, the sums as AdjSum, every atomic in FP64.  The
// FP64 pipe bounds it, so a warp keeps an instance's constants and Omega sums over
// all its targets (256^2, 32 + 32 samples: 512 -> 230 us a step, with one sum, atomic,
// root and quotient a target before).
template <bool F32>
__global__ void __launch_bounds__(256) k_adj_terms(AdjArgs a) {
    using R_ = typename std::conditional<F32, float, double>::type;
    const int lane = threadIdx.x & 31;
    const long warp = (long(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const long nwarps = (long(gridDim.x) * blockDim.x) >> 5;
    const int Q = a.N1 + a.N2;
    const double w1 = double(a.N1) / Q, w2 = double(a.N2) / Q, inv = 1.0 / Q;
    const R_* fg;
    if constexpr (F32) fg = a.fg32;
    else fg = a.fg;
    // what the warp's targets of one instance share: its constants and its sums
    int cur = -1;
    R_ rad = R_(0), w2a = R_(0), cum[2] = {R_(0), R_(0)}, icum[2] = {R_(0), R_(0)};
    AdjSum<F32> dca[2], csa[2];
    auto flush = [&]() {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const double dcs = warp_sum_d(dca[s].value());
            if (lane == 0 && dcs != 0.0) atomicAdd(&a.dcum[2 * cur + s], dcs);
            if (a.gsc) {
                const double css = warp_sum_d(csa[s].value());
                if (lane == 0 && css != 0.0) atomicAdd(&a.csum[2 * cur + s], css);
            }
            dca[s] = csa[s] = AdjSum<F32>();
        }
    };
    for (long tl = warp; tl < a.nt; tl += nwarps) {
        const long t = a.t0 + tl;
        const int ii = inst_of(a.mc, a.n_inst, t);
        const InstMC& I = a.mc[ii];
        if (ii != cur) {
            if (cur >= 0) flush();
            cur = ii;
            const double R = sqrt(double(I.Lx) * I.Lx + double(I.Ly) * I.Ly);   // as the FP64 path
            rad = R_(R);
            w2a = R_(w2 / (2.0 * kPiD * R));
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                cum[s] = R_(a.cum64[2 * ii + s]);
                icum[s] = R_(1.0 / a.cum64[2 * ii + s]);
            }
        }
        const float2 x = a.pos[t];
        const double mux = double(I.dt) * a.lam_next[2 * t], muy = double(I.dt) * a.lam_next[2 * t + 1];
        AdjSum<F32> ltx, lty;
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const double sg = (s == 0 ? inv : -inv);
            const R_ vx = R_(mux * sg), vy = R_(muy * sg);
            const long base = (tl * 2 + s) * Q;
            for (int j = lane; j < Q; j += 32) {
                const long sid = base + j;
                R_ gxx, gxy, df, dc, cv;
                mis_term_adj<R_>(I.law, x, a.ys[sid], fg[3 * sid], R_(w1), w2a, cum[s], icum[s], rad, I, vx, vy, gxx,
                                 gxy, df, dc, cv);
                const R_ fx = df * fg[3 * sid + 1], fy = df * fg[3 * sid + 2];   // dc/dy = -dc/dx|_f + dc/df grad f
                ltx.add(gxx);
                lty.add(gxy);
                if (j >= a.N1) {
                    ltx.add(-gxx);
                    ltx.add(fx);
                    lty.add(-gxy);
                    lty.add(fy);
                } else {
                    const double dyx = double(fx) - double(gxx), dyy = double(fy) - double(gxy);
                    const int p = a.src[sid];
                    if (p >= 0 && (dyx != 0.0 || dyy != 0.0)) {
                        atomicAdd(&a.lam[2 * p], dyx);
                        atomicAdd(&a.lam[2 * p + 1], dyy);
                    }
                    if (a.gsc && p >= 0 && cv != R_(0)) {
                        atomicAdd(&a.gsc[p], double(cv));
                        csa[s].add(cv);
                    }
                }
                a.as[sid] = double(df);
                dca[s].add(dc);
            }
        }
        const double lx = warp_sum_d(ltx.value()), ly = warp_sum_d(lty.value());
        if (lane == 0) {
            atomicAdd(&a.lam[2 * t], lx);
            atomicAdd(&a.lam[2 * t + 1], ly);
        }
    }
    if (cur >= 0) flush();
}

// The transposed sums (by grid slot) onto the particles: dL/domega through the
// strength, lambda through the position (the weight |omega| of each particle's
// kernel).  Each particle holds at most one slot (sign-split sets).
__global__ void k_adj_sources(const float* __restrict__ omega, const uint32_t* __restrict__ perm,
                              const uint32_t* __restrict__ cstart, uint32_t nbins, long n,
                              const double* __restrict__ dual, double* __restrict__ lam, double* __restrict__ gom) {
    const long nv = min(long(cstart[nbins]), n);
    for (long p = long(blockIdx.x) * blockDim.x + threadIdx.x; p < nv; p += long(gridDim.x) * blockDim.x) {
        const uint32_t i = perm[p];
        const float w = omega[i];
        if (w == 0.f) continue;
        const double aw = fabs(double(w));
        gom[i] += (w > 0.f ? 1.0 : -1.0) * dual[3 * p];
        lam[2 * i] += aw * dual[3 * p + 1];
        lam[2 * i + 1] += aw * dual[3 * p + 2];
    }
}

// Omega terms, and (score) the score-function term of the discrete branch-1
// draw P(I = J) = |omega_J| / Omega_s: d log P(I)/d omega_J =
// sgn(omega_J) (delta_IJ / |omega_J| - 1 / Omega_s), weighted by each sample's c.
__global__ void k_adj_cum(const InstMC* __restrict__ mc, int n_inst, const float* __restrict__ omega, long n,
                          const double* __restrict__ dcum, const double* __restrict__ cum64,
                          const double* __restrict__ gsc, const double* __restrict__ csum,
                          double* __restrict__ gom) {
    for (long i = long(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += long(gridDim.x) * blockDim.x) {
        const float w = omega[i];
        if (w == 0.f) continue;
        const int ii = inst_of(mc, n_inst, i);
        const int s = w > 0.f ? 0 : 1;
        const double sg = w > 0.f ? 1.0 : -1.0;
        const double f9 = mc[ii].periodic ? 9.0 : 1.0;
        double g = f9 * dcum[2 * ii + s];
        if (gsc) g += gsc[i] / fabs(double(w)) - csum[2 * ii + s] / (cum64[2 * ii + s] / f9);
        gom[i] += sg * g;
    }
}

// Adjoint working set (allocated on first use): per chunk of samples the
// source index, value + gradient (room for FP64; FP32 on the FP32 path) and FP64
// dc/df; per particle the transposed sums (by grid slot), two lambda buffers and
// dL/domega.
struct AdjBufs {
    int* src;
    double* fg;
    double* as;
    double* dual_out;
    double* lam[2];
    double* gom;
    double* dcum;
    double* gsc;
    double* csum;
};

int adj_bufs(vpmc_sim* s, AdjBufs* A) {
    const long ns = s->chunk_targets * 2 * samples_per(s);
    auto carve = [&](Carver& c) {
        A->src = c.take<int>(size_t(ns));
        A->fg = c.take<double>(3 * size_t(ns));
        A->as = c.take<double>(size_t(ns));
        A->dual_out = c.take<double>(3 * size_t(s->N));
        A->lam[0] = c.take<double>(2 * size_t(s->N));
        A->lam[1] = c.take<double>(2 * size_t(s->N));
        A->gom = c.take<double>(size_t(s->N));
        A->dcum = c.take<double>(2 * size_t(s->n_inst));
        A->gsc = c.take<double>(size_t(s->N));
        A->csum = c.take<double>(2 * size_t(s->n_inst));
    };
    Carver dry;
    carve(dry);
    VPMC_TRY(s->adj.reserve(dry.off));
    Carver c{static_cast<char*>(s->adj.p), 0};
    carve(c);
    return VPMC_OK;
}

// lam_out = lam_in + (dX'/dX)^T lam_in; gom += (dX'/domega)^T lam_in, at the
// state in s->pos with the step counter already on the device.
int adjoint_step(vpmc_sim* s, AdjBufs& A, const double* lam_in, double* lam_out, bool score) {
    vpmc_context* ctx = s->ctx;
    cudaStream_t st = ctx->stream;
    VPMC_TRY(grid_build(ctx, s->g, s->pos, s->omega, SET_SIGN_SPLIT));
    VPMC_CUDA(cudaMemcpyAsync(lam_out, lam_in, 2 * sizeof(double) * size_t(s->N), cudaMemcpyDeviceToDevice, st));
    VPMC_CUDA(cudaMemsetAsync(A.dcum, 0, 2 * sizeof(double) * size_t(s->n_inst), st));
    if (score) {
        VPMC_CUDA(cudaMemsetAsync(A.gsc, 0, sizeof(double) * size_t(s->N), st));
        VPMC_CUDA(cudaMemsetAsync(A.csum, 0, 2 * sizeof(double) * size_t(s->n_inst), st));
    }
    const bool unb = s->mc[0].law == VPMC_LAW_UNBIASED;
    const long Q = samples_per(s);
    for (long t0 = 0; t0 < s->N; t0 += s->chunk_targets) {
        const long nt = std::min(s->chunk_targets, s->N - t0);
        const long ns = nt * 2 * Q;
        const bool f32 = s->precision == 32;
        float* const fg32 = reinterpret_cast<float*>(A.fg);
        VPMC_TRY(clear_counts(ctx, s->q));
        GenArgs ga{s->d_mc, s->n_inst, s->g.inst, s->pos, nullptr, nullptr, s->sub, s->cdf, s->guide, s->jit, s->d_step, t0,
                   nt, s->N1, s->N2, 1, A.src, s->ys, s->q.qbin, s->q.qcount, s->q.qsub, s->q.qrank, f32 ? fg32 : nullptr, f32 ? nullptr : A.fg, 3};
        VPMC_TRY(launch_gen(st, ga));
        // f and grad f at every sample
        // (FP64 pairs: the forward's items, half-full where whole ones leave the device idle:
        // 32^2 particles, h_w 4 spacings, 8 + 8 samples, two steps and back 5.6 -> 3.9 ms)
        VPMC_TRY(place_samples(ctx, s->g, s->q, s->ys, ns, s->it, f32 ? query_chunk(4) : s->chunk64));
        EvalLaunch L;
        // field values and gradients at the samples: the FP32 path's adjoint sums
        // its pairs in FP32 (its terms read them in FP32; the candidates are the
        // particles in grid order, so the sums are fixed-order), the FP64 path's in FP64
        L.mode = unb ? (f32 ? EVAL_GRAD9_32 : EVAL_GRAD9_64) : (f32 ? EVAL_GRAD32 : EVAL_GRAD64);
        L.qpt = 4;
        L.out_f32 = fg32;
        L.out_f64 = A.fg;
        VPMC_TRY(launch_eval(ctx, s->g, s->q.qrec, s->it, L));
        AdjArgs aa{s->d_mc, s->n_inst, s->pos, s->ys, A.fg, fg32, A.src, s->cum64, t0, nt, s->N1, s->N2, lam_in, lam_out,
                   A.as, A.dcum, score ? A.gsc : nullptr, A.csum};
        // resident CTAs only: each warp keeps its sums over several targets
        int per_sm = 0;
        VPMC_CUDA(f32 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_adj_terms<true>, 256, 0)
                      : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_adj_terms<false>, 256, 0));
        const int terms_grid = std::min(blocks_for(nt * 32), ctx->sm_count * std::max(per_sm, 1));
        if (f32) VPMC_LAUNCH(k_adj_terms<true>, terms_grid, 256, 0, st, aa);
        else VPMC_LAUNCH(k_adj_terms<false>, terms_grid, 256, 0, st, aa);
        // transposed sums from the sample side: the same items, each sample
        // weighted by its dc/df, every in-support (sample, particle) pair adding
        // a_s W and a_s dW/dx_p to the particle's slot
        VPMC_CUDA(cudaMemsetAsync(s->it.counter, 0, sizeof(uint32_t), st));
        VPMC_CUDA(cudaMemsetAsync(A.dual_out, 0, 3 * sizeof(double) * size_t(s->N), st));
        EvalLaunch D;
        D.mode = unb ? (f32 ? EVAL_SCAT9_32 : EVAL_SCAT9_64) : (f32 ? EVAL_SCAT32 : EVAL_SCAT64);
        D.qpt = 4;
        D.out_f64 = A.dual_out;
        D.qweight = A.as;
        VPMC_TRY(launch_eval(ctx, s->g, s->q.qrec, s->it, D));
        VPMC_LAUNCH(k_adj_sources, blocks_for(s->N), 256, 0, st, s->omega, s->g.perm, s->g.cstart,
                    uint32_t(s->g.nbins), s->N, A.dual_out, lam_out, A.gom);
    }
    VPMC_LAUNCH(k_adj_cum, blocks_for(s->N), 256, 0, st, s->d_mc, s->n_inst, s->omega, s->N, A.dcum, s->cum64,
                score ? A.gsc : nullptr, A.csum, A.gom);
    return VPMC_OK;
}

}  // namespace
}  // namespace vpmc

using namespace vpmc;
using namespace vpmc::sim;

extern "C" {

int vpmc_sim_record(vpmc_sim* s, int nsteps, int k_ckpt) {
    if (!s || nsteps < 1 || k_ckpt < 1) return VPMC_ERR_INVALID;
    if (s->deform) return VPMC_ERR_UNSUPPORTED;   // the adjoint covers the plain method
    if (s->t_begin != 0 || s->t_end != s->N) return VPMC_ERR_UNSUPPORTED;   // and whole simulations, not shards
    VPMC_CUDA(cudaSetDevice(s->ctx->device));
    if (!s->prepared) VPMC_TRY(vpmc_sim_prepare(s));
    cudaStream_t st = s->ctx->stream;
    const long nck = (nsteps + k_ckpt - 1) / k_ckpt + 1;   // X_0, X_k, ..., and X_T
    VPMC_TRY(s->ckpt.reserve(sizeof(float2) * size_t(s->N) * size_t(nck)));
    float2* ck = static_cast<float2*>(s->ckpt.p);
    s->rec_steps = nsteps;
    s->rec_k = k_ckpt;
    s->rec_step0 = s->step;
    for (int n = 0; n < nsteps; ++n) {
        if (n % k_ckpt == 0)
            VPMC_CUDA(cudaMemcpyAsync(ck + size_t(n / k_ckpt) * s->N, s->pos, sizeof(float2) * size_t(s->N),
                                      cudaMemcpyDeviceToDevice, st));
        VPMC_TRY(run_pass(s, true, 1));
    }
    VPMC_CUDA(cudaMemcpyAsync(ck + size_t(nck - 1) * s->N, s->pos, sizeof(float2) * size_t(s->N),
                              cudaMemcpyDeviceToDevice, st));
    return vpmc_context_sync(s->ctx);
}

int vpmc_sim_adjoint(vpmc_sim* s, const double* dL_dXT, double* dL_dX0, double* dL_domega, int flags) {
    if (!s || !dL_dXT || !dL_dX0 || !dL_domega) return VPMC_ERR_INVALID;
    if (s->rec_steps < 1) return VPMC_ERR_INVALID;   // vpmc_sim_record first
    if (s->deform || s->t_begin != 0 || s->t_end != s->N) return VPMC_ERR_UNSUPPORTED;
    vpmc_context* ctx = s->ctx;
    VPMC_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    s->ys_t0 = -1;   // the adjoint redraws samples into the sample buffer
    s->ys_nt = 0;
    AdjBufs A;
    VPMC_TRY(adj_bufs(s, &A));
    const int T = s->rec_steps, k = s->rec_k;
    const long nck = (T + k - 1) / k + 1;
    float2* ck = static_cast<float2*>(s->ckpt.p);
    VPMC_TRY(s->seg.reserve(sizeof(float2) * size_t(s->N) * size_t(k)));
    float2* seg = static_cast<float2*>(s->seg.p);
    VPMC_CUDA(cudaMemcpyAsync(A.lam[0], dL_dXT, 2 * sizeof(double) * size_t(s->N), cudaMemcpyDeviceToDevice, st));
    VPMC_CUDA(cudaMemsetAsync(A.gom, 0, sizeof(double) * size_t(s->N), st));
    int cur = 0;
    for (long sg = nck - 2; sg >= 0; --sg) {
        const int n0 = int(sg) * k, n1 = std::min(T, n0 + k);
        // recompute the segment's states from its checkpoint (bitwise the forward's)
        VPMC_CUDA(cudaMemcpyAsync(s->pos, ck + size_t(sg) * s->N, sizeof(float2) * size_t(s->N),
                                  cudaMemcpyDeviceToDevice, st));
        VPMC_TRY(set_step_counter(s, s->rec_step0 + uint64_t(n0)));
        for (int n = n0; n < n1; ++n) {
            VPMC_CUDA(cudaMemcpyAsync(seg + size_t(n - n0) * s->N, s->pos, sizeof(float2) * size_t(s->N),
                                      cudaMemcpyDeviceToDevice, st));
            if (n + 1 < n1) VPMC_TRY(run_pass(s, true, 1));
        }
        for (int n = n1 - 1; n >= n0; --n) {
            VPMC_CUDA(cudaMemcpyAsync(s->pos, seg + size_t(n - n0) * s->N, sizeof(float2) * size_t(s->N),
                                      cudaMemcpyDeviceToDevice, st));
            VPMC_TRY(set_step_counter(s, s->rec_step0 + uint64_t(n)));
            VPMC_TRY(adjoint_step(s, A, A.lam[cur], A.lam[cur ^ 1], (flags & VPMC_ADJ_SCORE) != 0));
            cur ^= 1;
        }
    }
    VPMC_CUDA(cudaMemcpyAsync(dL_dX0, A.lam[cur], 2 * sizeof(double) * size_t(s->N), cudaMemcpyDeviceToDevice, st));
    VPMC_CUDA(cudaMemcpyAsync(dL_domega, A.gom, sizeof(double) * size_t(s->N), cudaMemcpyDeviceToDevice, st));
    // back to the recorded final state
    VPMC_CUDA(cudaMemcpyAsync(s->pos, ck + size_t(nck - 1) * s->N, sizeof(float2) * size_t(s->N),
                              cudaMemcpyDeviceToDevice, st));
    VPMC_TRY(set_step_counter(s, s->rec_step0 + uint64_t(T)));
    return vpmc_context_sync(ctx);
}

}  // extern "C"
