// vpmc_rbf.cu -- the RBF strength fits: conjugate gradients (the reference's
// conjugate_gradient_rbf, src/cuda/cg_rbf_init.cu:53-116) and MINRES on the
// matrix A_ij = W(|x_i - x_j|), and the matrix-free product (Ax_cuda,
// src/cuda/cg_rbf_init.cu:33-50).
//
// A solve applies the same matrix every iteration, and forming one FP64 kernel
// value takes ~20 instructions of a pipe with 2 lanes a clock and SM, so a
// solve forms the values once and keeps them for its iterations (12 bytes a
// pair, up to kMaxMatrixBytes; beyond, every product forms them again).  The
// scalars of an iteration stay on the device: each kernel sums the previous
// one's partial dots itself, so an iteration is three launches and the host
// only looks at the state every few iterations.  (192^2 particles, h_w = 8
// spacings, 7 MINRES iterations to 5e-3: 27.0 -> 1.11 ms.)
#include <algorithm>
#include <cmath>

#include "vpmc_work.cuh"

namespace vpmc {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr size_t kMaxMatrixBytes = size_t(4) << 30;
constexpr size_t kKeepMatrixBytes = size_t(512) << 20;   // a larger matrix is given back after the solve
constexpr int kPartMax = 2048;                           // partial sums a reduction reads (every CTA reads them all)

__global__ void k_self_queries(const Cand* __restrict__ cand, const uint32_t* __restrict__ start, long n,
                               uint32_t nbins, QRec* __restrict__ q) {
    const long nv = start[nbins];
    for (long p = long(blockIdx.x) * blockDim.x + threadIdx.x; p < nv && p < n; p += long(gridDim.x) * blockDim.x) {
        const Cand c = cand[p];
        q[p] = QRec{c.x, c.y, uint32_t(p), (2u) | (2u << 3)};
    }
}

template <typename T>
__global__ void k_gather_to_sorted(const T* __restrict__ x, const uint32_t* __restrict__ perm, long n,
                                   double* __restrict__ xs) {
    for (long p = long(blockIdx.x) * blockDim.x + threadIdx.x; p < n; p += long(gridDim.x) * blockDim.x)
        xs[p] = double(x[perm[p]]);
}

__global__ void k_scatter_from_sorted(const double* __restrict__ xs, const uint32_t* __restrict__ perm, long n,
                                      float* __restrict__ x) {
    for (long p = long(blockIdx.x) * blockDim.x + threadIdx.x; p < n; p += long(gridDim.x) * blockDim.x)
        x[perm[p]] = float(xs[p]);
}

// ------------------------------------------------------------ the kept matrix
// Rows are the particles in grid order, 32 consecutive rows a slice; entry e of
// lane l of slice s is at (off[s] + e) 32 + l, so a warp reads its 32 values of
// one entry in one line each.  A slice is as long as its longest row; the other
// rows end in zero values at their own index.
struct RbfMatrix {
    long n = 0, nslices = 0;
    uint32_t* len = nullptr;      // per slice: entries
    uint32_t* off = nullptr;      // per slice: first entry (in units of 32)
    unsigned long long* cursor = nullptr;   // [0]: sum of len, [1]: entries placed
    unsigned long long room = 0;            // entries there is memory for (in units of 32)
    uint32_t* idx = nullptr;
    double* val = nullptr;
};

// Visit every candidate of lane's row in the order of the walk, candidates
// part, part + kWarps, ... of each run (the walk is the evaluation kernel's).
template <typename Fn>
__device__ __forceinline__ void visit_row(const GridInst& G, const uint32_t* __restrict__ start, float px, float py,
                                          int part, Fn&& fn) {
    const int cx = min(max(floor_int(px * G.inv_sx), 0), G.gx - 1);
    const int cy = min(max(floor_int(py * G.inv_sy), 0), G.gy - 1);
    for (int col = 0; col <= 2 * G.k; ++col) {
        int gxx, sxi, r0[2], r1[2], syi[2];
        walk_column(G, cx, cy, 1, col, gxx, sxi, r0, r1, syi);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (r0[h] > r1[h]) continue;
            const uint32_t b0 = uint32_t(G.bin_base) + uint32_t(gxx * G.gy + r0[h]);
            const uint32_t c1 = start[b0 + uint32_t(r1[h] - r0[h]) + 1];
            const float qx = __fsub_rn(px, float(sxi) * G.Lx), qy = __fsub_rn(py, float(syi[h]) * G.Ly);
            for (uint32_t c = start[b0] + uint32_t(part); c < c1; c += kWarps) fn(c, qx, qy);
        }
    }
}

// Whether candidate c may be within the support of (qx, qy) (as the matrix-free
// product tests it; a pair beyond the support then has a zero value).
__device__ __forceinline__ bool near_pair(const Cand& c, float qx, float qy, float lim) {
    const float dx = __fsub_rn(c.x, qx), dy = __fsub_rn(c.y, qy);
    return __fmaf_rn(dx, dx, __fmul_rn(dy, dy)) < lim;
}

// One CTA a slice; its warps share each row's candidates.  Without kFill the
// entries the slice needs are counted; with it the indices are written (a row's
// entries ordered by warp, then by the walk: fixed), the slice placed where a
// counter stands (the place has no influence on any value).
template <bool kFill>
__global__ void __launch_bounds__(kThreads) k_rbf_rows(const GridInst* __restrict__ inst,
                                                       const uint32_t* __restrict__ start,
                                                       const Cand* __restrict__ cand, long n, RbfMatrix A,
                                                       unsigned* __restrict__ flags) {
    __shared__ uint32_t cnt[kWarps][32];
    __shared__ uint32_t s_off;
    const GridInst G = inst[0];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const float lim = G.hw * G.hw * 1.0001f;
    for (long s = blockIdx.x; s < A.nslices; s += gridDim.x) {
        const long row = s * 32 + lane;
        const bool live = row < n;
        const float px = live ? cand[row].x : 0.f, py = live ? cand[row].y : 0.f;
        uint32_t c = 0;
        if (live)
            visit_row(G, start, px, py, w,
                      [&](uint32_t j, float qx, float qy) { c += near_pair(cand[j], qx, qy, lim) ? 1u : 0u; });
        cnt[w][lane] = c;
        __syncthreads();
        uint32_t before = 0, total = 0;
#pragma unroll
        for (int i = 0; i < kWarps; ++i) {
            if (i < w) before += cnt[i][lane];
            total += cnt[i][lane];
        }
        uint32_t most = total;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
        if (threadIdx.x == 0) {
            if (kFill) {
                const unsigned long long at = atomicAdd(&A.cursor[1], (unsigned long long)most);
                const bool fits = at + most <= A.room;   // the counting pass sized it: always
                if (!fits) atomicOr(flags, FLAG_INTERNAL);
                s_off = fits ? uint32_t(at) : 0xffffffffu;
                A.off[s] = fits ? uint32_t(at) : 0u;
                A.len[s] = fits ? most : 0u;
            } else {
                atomicAdd(&A.cursor[0], (unsigned long long)most);
            }
        }
        __syncthreads();
        if (kFill && s_off != 0xffffffffu) {
            uint32_t* at = A.idx + size_t(s_off) * 32 + lane;
            uint32_t e = before;
            const uint32_t end = before + c;
            if (live)
                visit_row(G, start, px, py, w, [&](uint32_t j, float qx, float qy) {
                    if (near_pair(cand[j], qx, qy, lim) && e < end) at[size_t(e++) * 32] = j;
                });
            for (; e < end; ++e) at[size_t(e) * 32] = 0xffffffffu;
            for (uint32_t k = total + w; k < most; k += kWarps) at[size_t(k) * 32] = 0xffffffffu;
        }
        __syncthreads();
    }
}

// The values, FP64, each entry on its own lane, so no lane waits for a pair
// outside the support.  They are the numbers spline_w_d gives (the matrix-free
// product's), in 26 FP64 instructions instead of ~35: the root and the quotient
// r / h come from an estimate (the hardware's, 1 / h) by fused residual
// corrections (Markstein, IBM J. Res. Dev. 34, 1990); over 2^30 distances, across the
// pieces, at the knots and down to 2^-400 h, root, quotient and value had the bits of
// sqrt, of the division and of spline_w_d.
// FP64-pipe bound (192^2, h_w = 8: 7.8 M entries, 0.47 ms).
__global__ void __launch_bounds__(kThreads) k_rbf_values(const GridInst* __restrict__ inst,
                                                         const Cand* __restrict__ cand, long n, RbfMatrix A) {
    const GridInst G = inst[0];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const double hw = double(G.hw), ih = 1.0 / hw, sigma = 40.0 / (7.0 * kPiD * hw * hw);
    const float hx = 0.5f * G.Lx, hy = 0.5f * G.Ly;
    for (long s = blockIdx.x; s < A.nslices; s += gridDim.x) {
        const long row = s * 32 + lane;
        const bool live = row < n;
        const float px = live ? cand[row].x : 0.f, py = live ? cand[row].y : 0.f;
        const double pxd = px, pyd = py;
        const uint32_t len = A.len[s];
        const size_t base = size_t(A.off[s]) * 32 + lane;
        for (uint32_t e = w; e < len; e += kWarps) {
            const uint32_t j = A.idx[base + size_t(e) * 32];
            double v = 0.0;
            if (j != 0xffffffffu) {
                const float cx = cand[j].x, cy = cand[j].y;
                double ox = pxd, oy = pyd;
                if (G.periodic) {   // the image within the support (the support is below half a period)
                    if (fabsf(cx - px) > hx) ox += double(cx > px ? G.Lx : -G.Lx);
                    if (fabsf(cy - py) > hy) oy += double(cy > py ? G.Ly : -G.Ly);
                }
                const double dx = double(cx) - ox, dy = double(cy) - oy;
                const double r2 = dx * dx + dy * dy;
                double y;
                asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(r2));
                const double d = fma(-(r2 * y), y, 1.0);
                y = fma(y * d, fma(d, 0.375, 0.5), y);
                const double g = r2 * y;
                const double r = fma(fma(-g, g, r2), 0.5 * y, g);
                double q = r * ih;
                q = fma(fma(-q, hw, r), ih, q);
                const double t = 1.0 - q;
                const double inner = sigma * (6.0 * (q * q * q - q * q) + 1.0), outer = sigma * 2.0 * t * t * t;
                // ordered by the bits (q >= 0); r2 = 0 (and below the estimate's range) gives q = NaN: the centre
                const long long qb = __double_as_longlong(q);
                v = qb <= 0x3fe0000000000000ll ? inner : qb < 0x3ff0000000000000ll ? outer : 0.0;
                if (__double2hiint(r2) < 0x00200000) v = sigma;
            } else {
                A.idx[base + size_t(e) * 32] = live ? uint32_t(row) : 0u;
            }
            A.val[base + size_t(e) * 32] = v;
        }
    }
}

// ------------------------------------------------- solver state and reductions
// Device-resident scalars of a solve.
struct SolveState {
    double bnorm, tol;
    double beta, eta, c0, c1, s0, s1;   // MINRES: Lanczos beta, residual norm with sign, the last two rotations
    double rr;                          // CG: r . r
    double res;                         // CG: residual norm / bnorm
    double alpha;
    double ee;                          // true residual norm^2
    int it, max_iter, done;
};

// Sum of part[0..np) in a fixed order, the same in every thread of the CTA.
__device__ __forceinline__ double sum_parts(const double* __restrict__ part, int np) {
    __shared__ double sh[kWarps];
    double v = 0.0;
    for (int i = threadIdx.x; i < np; i += kThreads) v += part[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();   // sh may still be read from the previous sum
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
#pragma unroll
    for (int i = 0; i < kWarps; ++i) t += sh[i];
    return t;
}

// The CTA's sum of v, written to part[blockIdx.x].
__device__ __forceinline__ void write_part(double v, double* __restrict__ part) {
    __shared__ double sh[kWarps];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
#pragma unroll
        for (int i = 0; i < kWarps; ++i) t += sh[i];
        part[blockIdx.x] = t;
    }
}

// y = A x with the kept matrix, and the partial sums of x . y.  The eight warps
// of a CTA take a slice's entries in turn (four sums a warp in flight) and their
// sums are added in warp order.
// Bound by reading the matrix: 12 bytes an entry (192^2, h_w = 8: 94 MB in
// 20.7 us from a cold cache).
__global__ void __launch_bounds__(kThreads) k_rbf_product(RbfMatrix A, const double* __restrict__ x,
                                                          double* __restrict__ y, double* __restrict__ part,
                                                          const SolveState* __restrict__ st) {
    __shared__ double red[2][kWarps][32];
    if (st && st->done) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double dot = 0.0;
    int buf = 0;
    for (long s = blockIdx.x; s < A.nslices; s += gridDim.x, buf ^= 1) {
        const uint32_t len = A.len[s];
        const size_t base = size_t(A.off[s]) * 32 + lane;
        const uint32_t* __restrict__ idx = A.idx + base;
        const double* __restrict__ val = A.val + base;
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        uint32_t e = w;
        for (; e + 3 * kWarps < len; e += 4 * kWarps) {
            uint32_t j[4];
            double v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                j[k] = __ldcs(idx + size_t(e + k * kWarps) * 32);
                v[k] = __ldcs(val + size_t(e + k * kWarps) * 32);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[k] = fma(v[k], x[j[k]], acc[k]);
        }
        for (; e < len; e += kWarps)
            acc[0] = fma(__ldcs(val + size_t(e) * 32), x[__ldcs(idx + size_t(e) * 32)], acc[0]);
        red[buf][w][lane] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
        __syncthreads();   // one barrier a slice: the next slice writes the other buffer
        if (w == 0) {
            double t = 0.0;
#pragma unroll
            for (int i = 0; i < kWarps; ++i) t += red[buf][i][lane];
            const long row = s * 32 + lane;
            if (row < A.n) {
                y[row] = t;
                dot = fma(x[row], t, dot);
            }
        }
    }
    if (part) {
        __syncthreads();
        write_part(dot, part);
    }
}

// Partial sums of x . y (the matrix-free product's dot).
__global__ void __launch_bounds__(kThreads) k_rbf_dot(const double* __restrict__ x, const double* __restrict__ y,
                                                      long n, double* __restrict__ part,
                                                      const SolveState* __restrict__ st) {
    if (st && st->done) return;
    double s = 0.0;
    for (long i = long(blockIdx.x) * kThreads + threadIdx.x; i < n; i += long(gridDim.x) * kThreads)
        s = fma(x[i], y[i], s);
    write_part(s, part);
}

__global__ void k_scale(const double* __restrict__ a, long n, double s, double* __restrict__ out) {
    for (long i = long(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += long(gridDim.x) * blockDim.x)
        out[i] = s * a[i];
}

// r = b - Ax with the partial sums of b . b (when pb) and r . r.
__global__ void __launch_bounds__(kThreads) k_residual(const double* __restrict__ b, const double* __restrict__ Ax,
                                                       long n, double* __restrict__ r, double* __restrict__ pb,
                                                       double* __restrict__ pr) {
    double sb = 0.0, sr = 0.0;
    for (long i = long(blockIdx.x) * kThreads + threadIdx.x; i < n; i += long(gridDim.x) * kThreads) {
        const double v = b[i] - Ax[i];
        r[i] = v;
        sb = fma(b[i], b[i], sb);
        sr = fma(v, v, sr);
    }
    if (pb) {
        write_part(sb, pb);
        __syncthreads();
    }
    write_part(sr, pr);
}

__global__ void __launch_bounds__(kThreads) k_true_residual(const double* __restrict__ pr, int np, SolveState* st) {
    const double t = sum_parts(pr, np);
    if (threadIdx.x == 0) st->ee = t;
}

// --------------------------------------------------------------------- MINRES
// (Paige & Saunders, SIAM J. Numer. Anal. 12, 1975): Lanczos vectors, one Givens
// rotation an iteration, the residual norm |eta| decreasing monotonically.
// Unlike CG it needs no definiteness, which the RBF matrix lacks (its spline
// symbol is negative at high wavenumbers, with eigenvalues near zero on both sides).
// v = r / |r|, the other vectors zero, the state of iteration 0.
__global__ void __launch_bounds__(kThreads) k_minres_begin(const double* __restrict__ r, const double* __restrict__ pb,
                                                           const double* __restrict__ pr, int np, long n, double tol,
                                                           int max_iter, double* __restrict__ v,
                                                           double* __restrict__ v_old, double* __restrict__ w,
                                                           double* __restrict__ w_old, SolveState* __restrict__ st) {
    const double bnorm = sqrt(sum_parts(pb, np)), beta = sqrt(sum_parts(pr, np));
    const double inv = beta > 0.0 ? 1.0 / beta : 0.0;
    for (long i = long(blockIdx.x) * kThreads + threadIdx.x; i < n; i += long(gridDim.x) * kThreads) {
        v[i] = r[i] * inv;
        v_old[i] = w[i] = w_old[i] = 0.0;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        SolveState s{};
        s.bnorm = bnorm;
        s.tol = tol;
        s.beta = beta;
        s.eta = beta;
        s.c0 = s.c1 = 1.0;
        s.max_iter = max_iter;
        s.done = !(bnorm > 0.0 && beta > 0.0 && max_iter > 0 && fabs(beta) >= tol * bnorm);
        st[0] = st[1] = s;
    }
}

// u = Av - alpha v - beta v_old (the next Lanczos vector before normalisation)
__global__ void __launch_bounds__(kThreads) k_minres_u(double* __restrict__ u, const double* __restrict__ v,
                                                       const double* __restrict__ v_old, long n,
                                                       const double* __restrict__ pa, int npa,
                                                       const SolveState* __restrict__ st, double* __restrict__ pu) {
    if (st->done) return;
    const double alpha = sum_parts(pa, npa), beta = st->beta;
    double s = 0.0;
    for (long i = long(blockIdx.x) * kThreads + threadIdx.x; i < n; i += long(gridDim.x) * kThreads) {
        const double t = u[i] - alpha * v[i] - beta * v_old[i];
        u[i] = t;
        s = fma(t, t, s);
    }
    write_part(s, pu);
}

// The rotation, then w_new = (v - rho3 w_old - rho2 w) / rho1 (over w_old),
// x += c eta w_new, v_next = u / beta_n (over v_old); every CTA forms the scalars
// itself from `st`, CTA 0 writes the next state to `next`.
__global__ void __launch_bounds__(kThreads) k_minres_step(const double* __restrict__ u, const double* __restrict__ v,
                                                          double* __restrict__ v_old, const double* __restrict__ w,
                                                          double* __restrict__ w_old, double* __restrict__ x, long n,
                                                          const double* __restrict__ pa, int npa,
                                                          const double* __restrict__ pu, int npu,
                                                          const SolveState* __restrict__ st,
                                                          SolveState* __restrict__ next) {
    SolveState s = *st;
    if (s.done) {
        if (blockIdx.x == 0 && threadIdx.x == 0) *next = s;
        return;
    }
    const double alpha = sum_parts(pa, npa), beta_n = sqrt(sum_parts(pu, npu));
    const double delta = s.c1 * alpha - s.c0 * s.s1 * s.beta;
    const double rho1 = hypot(delta, beta_n);
    const double rho2 = s.s1 * alpha + s.c0 * s.c1 * s.beta;
    const double rho3 = s.s0 * s.beta;
    if (!(rho1 > 0.0) || !isfinite(rho1)) {
        s.done = 1;
        if (blockIdx.x == 0 && threadIdx.x == 0) *next = s;
        return;
    }
    s.c0 = s.c1;
    s.s0 = s.s1;
    s.c1 = delta / rho1;
    s.s1 = beta_n / rho1;
    const double c = s.c1 * s.eta, inv = beta_n > 0.0 ? 1.0 / beta_n : 0.0;
    for (long i = long(blockIdx.x) * kThreads + threadIdx.x; i < n; i += long(gridDim.x) * kThreads) {
        const double wn = (v[i] - rho3 * w_old[i] - rho2 * w[i]) / rho1;
        w_old[i] = wn;
        x[i] += c * wn;
        v_old[i] = u[i] * inv;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        s.eta = -s.s1 * s.eta;
        s.beta = beta_n;
        s.it += 1;
        // beta_n == 0: the Krylov space is invariant and x is exact
        s.done = beta_n == 0.0 || !(s.it < s.max_iter && fabs(s.eta) >= s.tol * s.bnorm);
        *next = s;
    }
}

// ------------------------------------------------------------------------- CG
__global__ void __launch_bounds__(kThreads) k_cg_begin(const double* __restrict__ r, const double* __restrict__ pb,
                                                       const double* __restrict__ pr, int np, long n, double tol,
                                                       int max_iter, double* __restrict__ p,
                                                       SolveState* __restrict__ st) {
    const double bnorm = sqrt(sum_parts(pb, np)), rr = sum_parts(pr, np);
    for (long i = long(blockIdx.x) * kThreads + threadIdx.x; i < n; i += long(gridDim.x) * kThreads) p[i] = r[i];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        SolveState s{};
        s.bnorm = bnorm;
        s.tol = tol;
        s.rr = rr;
        s.res = bnorm > 0.0 ? sqrt(rr) / bnorm : 0.0;
        s.max_iter = max_iter;
        s.done = !(max_iter > 0 && s.res >= tol && bnorm > 0.0);
        st[0] = st[1] = s;
    }
}

__global__ void __launch_bounds__(kThreads) k_cg_xr(double* __restrict__ x, double* __restrict__ r,
                                                    const double* __restrict__ p, const double* __restrict__ Ap, long n,
                                                    const double* __restrict__ pa, int npa,
                                                    const SolveState* __restrict__ st, double* __restrict__ pr) {
    if (st->done) return;
    const double pAp = sum_parts(pa, npa);
    if (pAp == 0.0 || !isfinite(pAp)) return;   // k_cg_p ends the solve
    const double alpha = st->rr / pAp;
    double s = 0.0;
    for (long i = long(blockIdx.x) * kThreads + threadIdx.x; i < n; i += long(gridDim.x) * kThreads) {
        x[i] += alpha * p[i];
        const double v = r[i] - alpha * Ap[i];
        r[i] = v;
        s = fma(v, v, s);
    }
    write_part(s, pr);
}

__global__ void __launch_bounds__(kThreads) k_cg_p(double* __restrict__ p, const double* __restrict__ r, long n,
                                                   const double* __restrict__ pa, int npa,
                                                   const double* __restrict__ pr, int npr,
                                                   const SolveState* __restrict__ st, SolveState* __restrict__ next) {
    SolveState s = *st;
    const double pAp = s.done ? 0.0 : sum_parts(pa, npa);
    if (s.done || pAp == 0.0 || !isfinite(pAp)) {
        s.done = 1;
        if (blockIdx.x == 0 && threadIdx.x == 0) *next = s;
        return;
    }
    const double rr = sum_parts(pr, npr), beta = rr / s.rr;
    s.it += 1;
    s.res = sqrt(rr) / s.bnorm;
    s.done = !(s.res >= s.tol && s.it < s.max_iter);
    if (!s.done)
        for (long i = long(blockIdx.x) * kThreads + threadIdx.x; i < n; i += long(gridDim.x) * kThreads)
            p[i] = r[i] + beta * p[i];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        s.rr = rr;
        *next = s;
    }
}

// ------------------------------------------------------------------ host side
struct Solver {
    Work w;
    RbfMatrix A;
    bool kept = false;
    long N = 0;
    int vgrid = 1, pgrid = 1;         // CTAs of the vector kernels / of the product
    double *pa = nullptr, *pb = nullptr, *pr = nullptr;
    SolveState* st = nullptr;         // two, written in turn
};

// y = A x (and the partial sums of x . y in s.pa when dot).
int product(vpmc_context* ctx, Solver& s, const double* x, double* y, bool dot, const SolveState* st) {
    if (s.kept) {
        VPMC_LAUNCH(k_rbf_product, s.pgrid, kThreads, 0, ctx->stream, s.A, x, y, dot ? s.pa : nullptr, st);
        return VPMC_OK;
    }
    VPMC_TRY(grid_set_weights_sorted(ctx, s.w.g, x, 1.0));
    EvalLaunch L;
    L.mode = EVAL_SPMV64;
    L.out_f64 = y;
    VPMC_CUDA(cudaMemsetAsync(s.w.it.counter, 0, sizeof(uint32_t), ctx->stream));
    VPMC_TRY(launch_eval(ctx, s.w.g, s.w.self, s.w.it, L));
    if (dot) VPMC_LAUNCH(k_rbf_dot, s.pgrid, kThreads, 0, ctx->stream, x, y, s.N, s.pa, st);
    return VPMC_OK;
}

// Grid, right-hand side, the matrix when it fits, x0 = b / W(0) (the reference's
// starting point), r = b - A x0 and the partial sums of b . b and r . r.
int begin(vpmc_context* ctx, Solver& s, int N, const float* pos, const float* b, const double* b64, float h_w, float Lx,
          float Ly, double* r) {
    cudaStream_t st = ctx->stream;
    Work& w = s.w;
    VPMC_TRY(grid_build(ctx, w.g, reinterpret_cast<const float2*>(pos), nullptr, SET_ONE_SIGNED));
    RbfMatrix& A = s.A;
    A.n = N;
    A.nslices = (long(N) + 31) / 32;
    const int grid = int(std::min<long>(A.nslices, 65535L * 8));
    VPMC_CUDA(cudaMemsetAsync(A.cursor, 0, 2 * sizeof(unsigned long long), st));
    // particles spread evenly have N pi h^2 / (Lx Ly) neighbours: a matrix far
    // from fitting by that is not counted
    const double even = double(N) * std::min(1.0, kPiD * h_w * h_w / (double(Lx) * Ly));
    // (a kept matrix has no staging wait to give up: a limit of 0 polls takes the products
    // that form the values, whose first wait then expires)
    if (ctx->wait_limit > 0 && double(N) * even * 12.0 <= 2.0 * double(kMaxMatrixBytes)) {
        VPMC_LAUNCH(k_rbf_rows<false>, grid, kThreads, 0, st, w.g.inst, w.g.cstart, w.g.cand, long(N), A, ctx->d_flags);
        unsigned long long total = 0;
        VPMC_CUDA(cudaMemcpyAsync(&total, A.cursor, sizeof(total), cudaMemcpyDeviceToHost, st));
        VPMC_CUDA(cudaStreamSynchronize(st));
        const size_t entries = size_t(total) * 32, bytes = entries * 12 + 1024;
        char* base = nullptr;
        if (total <= kMaxMatrixBytes / (32 * 12)) {
            const int rc = scratch(ctx, SLOT_MATRIX, bytes, &base);
            if (rc != VPMC_OK && rc != VPMC_ERR_NOMEM) return rc;
            s.kept = rc == VPMC_OK;   // without room the products form the values
        }
        if (s.kept) {
            Carver c{base, 0};
            A.val = c.take<double>(entries);
            A.idx = c.take<uint32_t>(entries);
            A.room = total;
            VPMC_LAUNCH(k_rbf_rows<true>, grid, kThreads, 0, st, w.g.inst, w.g.cstart, w.g.cand, long(N), A, ctx->d_flags);
            VPMC_LAUNCH(k_rbf_values, grid, kThreads, 0, st, w.g.inst, w.g.cand, long(N), A);
        }
    }
    if (!s.kept) {
        VPMC_LAUNCH(k_self_queries, work_blocks(N), 256, 0, st, w.g.cand, w.g.cstart, long(N), uint32_t(w.g.nbins),
                    w.self);
        VPMC_TRY(make_items(ctx, w.g, w.g.cstart, w.it, query_chunk(4), N));
    }
    double *bs = w.vec[0], *x = w.vec[1];
    if (b64) VPMC_LAUNCH(k_gather_to_sorted<double>, work_blocks(N), 256, 0, st, b64, w.g.perm, long(N), bs);
    else VPMC_LAUNCH(k_gather_to_sorted<float>, work_blocks(N), 256, 0, st, b, w.g.perm, long(N), bs);
    const double diag = spline_w_d(0.0, double(h_w));
    VPMC_LAUNCH(k_scale, work_blocks(N), 256, 0, st, bs, long(N), 1.0 / diag, x);
    VPMC_TRY(product(ctx, s, x, r, false, nullptr));
    VPMC_LAUNCH(k_residual, s.vgrid, kThreads, 0, st, bs, r, long(N), r, s.pb, s.pr);
    return VPMC_OK;
}

int solver_setup(vpmc_context* ctx, Solver& s, int N, float h_w, float Lx, float Ly, int periodic, int nvec) {
    // the solver's own arrays follow the grid's in one slot
    VPMC_TRY(setup_work(ctx, SLOT_CG, N, h_w, Lx, Ly, periodic, 0, nvec, &s.w));
    s.N = N;
    const long ns = (long(N) + 31) / 32;
    s.vgrid = int(std::max<long>(1, std::min<long>((long(N) + kThreads - 1) / kThreads, 4L * ctx->sm_count)));
    s.pgrid = int(std::max<long>(1, std::min<long>(ns, 8L * ctx->sm_count)));
    s.vgrid = std::min(s.vgrid, kPartMax);
    s.pgrid = std::min(s.pgrid, kPartMax);
    auto carve = [&](Carver& c) {
        s.A.len = c.take<uint32_t>(size_t(ns));
        s.A.off = c.take<uint32_t>(size_t(ns));
        s.A.cursor = c.take<unsigned long long>(2);
        s.pa = c.take<double>(kPartMax);
        s.pb = c.take<double>(kPartMax);
        s.pr = c.take<double>(kPartMax);
        s.st = c.take<SolveState>(2);
    };
    Carver dry;
    carve(dry);
    char* base = nullptr;
    VPMC_TRY(scratch(ctx, SLOT_SOLVE, dry.off, &base));
    Carver c{base, 0};
    carve(c);
    return VPMC_OK;
}

// Run `iteration(i)` (three launches; a finished solve makes them return at once)
// until the state says done.  The host looks at it after 4, 8, 12 and 16
// iterations, then after every 16; where a product forms its values (and could
// not return at once) before each one.
template <typename Fn>
int iterate(vpmc_context* ctx, Solver& s, SolveState* h, Fn&& iteration) {
    cudaStream_t st = ctx->stream;
    int i = 0;
    auto look = [&]() -> int {
        VPMC_CUDA(cudaMemcpyAsync(h, &s.st[i & 1], sizeof(*h), cudaMemcpyDeviceToHost, st));
        VPMC_CUDA(cudaStreamSynchronize(st));
        return VPMC_OK;
    };
    if (!s.kept) VPMC_TRY(look());
    while (!h->done) {
        const int batch = !s.kept ? 1 : i < 16 ? 4 : 16;
        for (int k = 0; k < batch; ++k, ++i) VPMC_TRY(iteration(i));
        VPMC_TRY(look());
    }
    return VPMC_OK;
}

// The true residual with one more product, the strengths back in the caller's
// order, and a matrix above kKeepMatrixBytes given back.
int finish(vpmc_context* ctx, Solver& s, double* x, double* u, float* omega_out, SolveState* h) {
    cudaStream_t st = ctx->stream;
    VPMC_TRY(product(ctx, s, x, u, false, nullptr));
    VPMC_LAUNCH(k_residual, s.vgrid, kThreads, 0, st, s.w.vec[0], u, s.N, u, static_cast<double*>(nullptr), s.pr);
    VPMC_LAUNCH(k_true_residual, 1, kThreads, 0, st, s.pr, s.vgrid, s.st);
    VPMC_LAUNCH(k_scatter_from_sorted, work_blocks(s.N), 256, 0, st, x, s.w.g.perm, s.N, omega_out);
    VPMC_CUDA(cudaMemcpyAsync(&h->ee, &s.st[0].ee, sizeof(double), cudaMemcpyDeviceToHost, st));
    VPMC_TRY(vpmc_context_sync(ctx));
    if (ctx->scratch[SLOT_MATRIX].bytes > kKeepMatrixBytes) ctx->scratch[SLOT_MATRIX].release();
    return VPMC_OK;
}

int cg_impl(vpmc_context* ctx, int N, const float* pos, const float* b, const double* b64, float* omega_out, float h_w,
            float Lx, float Ly, int periodic, double tol, int max_iter, double* info) {
    if (!ctx || N < 0 || !(h_w > 0.f) || !(Lx > 0.f) || !(Ly > 0.f) || max_iter < 0) return VPMC_ERR_INVALID;
    if (N == 0) {
        if (info) { info[0] = 0; info[1] = 0; info[2] = 0; }
        return VPMC_OK;
    }
    if (!pos || (!b && !b64) || !omega_out) return VPMC_ERR_INVALID;
    VPMC_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    Solver s;
    VPMC_TRY(solver_setup(ctx, s, N, h_w, Lx, Ly, periodic, 5));
    double *x = s.w.vec[1], *r = s.w.vec[2], *p = s.w.vec[3], *Ap = s.w.vec[4];
    VPMC_TRY(begin(ctx, s, N, pos, b, b64, h_w, Lx, Ly, r));
    VPMC_LAUNCH(k_cg_begin, s.vgrid, kThreads, 0, st, r, s.pb, s.pr, s.vgrid, long(N), tol, max_iter, p, s.st);
    SolveState h{};
    VPMC_TRY(iterate(ctx, s, &h, [&](int i) -> int {
        const SolveState* now = &s.st[i & 1];
        VPMC_TRY(product(ctx, s, p, Ap, true, now));
        VPMC_LAUNCH(k_cg_xr, s.vgrid, kThreads, 0, st, x, r, p, Ap, long(N), s.pa, s.pgrid, now, s.pr);
        VPMC_LAUNCH(k_cg_p, s.vgrid, kThreads, 0, st, p, r, long(N), s.pa, s.pgrid, s.pr, s.vgrid, now,
                    &s.st[(i + 1) & 1]);
        return VPMC_OK;
    }));
    VPMC_TRY(finish(ctx, s, x, Ap, omega_out, &h));
    if (info) {
        info[0] = h.it;
        info[1] = h.res;
        info[2] = h.bnorm > 0 ? std::sqrt(h.ee) / h.bnorm : 0.0;
    }
    return h.res < tol || h.bnorm == 0 ? VPMC_OK : VPMC_ERR_NOT_CONVERGED;
}

int minres_impl(vpmc_context* ctx, int N, const float* pos, const float* b, const double* b64, float* omega_out,
                float h_w, float Lx, float Ly, int periodic, double tol, int max_iter, double* info) {
    if (!ctx || N < 0 || !(h_w > 0.f) || !(Lx > 0.f) || !(Ly > 0.f) || max_iter < 0) return VPMC_ERR_INVALID;
    if (N == 0) {
        if (info) { info[0] = 0; info[1] = 0; info[2] = 0; }
        return VPMC_OK;
    }
    if (!pos || (!b && !b64) || !omega_out) return VPMC_ERR_INVALID;
    VPMC_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    Solver s;
    VPMC_TRY(solver_setup(ctx, s, N, h_w, Lx, Ly, periodic, 7));
    double* x = s.w.vec[1];
    double* v[2] = {s.w.vec[2], s.w.vec[3]};       // v, v_old in turn
    double* wv[2] = {s.w.vec[4], s.w.vec[5]};      // w, w_old in turn
    double* u = s.w.vec[6];
    VPMC_TRY(begin(ctx, s, N, pos, b, b64, h_w, Lx, Ly, u));
    VPMC_LAUNCH(k_minres_begin, s.vgrid, kThreads, 0, st, u, s.pb, s.pr, s.vgrid, long(N), tol, max_iter, v[0], v[1],
                wv[0], wv[1], s.st);
    SolveState h{};
    VPMC_TRY(iterate(ctx, s, &h, [&](int i) -> int {
        const SolveState* now = &s.st[i & 1];
        const int a = i & 1, o = a ^ 1;
        VPMC_TRY(product(ctx, s, v[a], u, true, now));
        VPMC_LAUNCH(k_minres_u, s.vgrid, kThreads, 0, st, u, v[a], v[o], long(N), s.pa, s.pgrid, now, s.pr);
        VPMC_LAUNCH(k_minres_step, s.vgrid, kThreads, 0, st, u, v[a], v[o], wv[a], wv[o], x, long(N), s.pa, s.pgrid,
                    s.pr, s.vgrid, now, &s.st[(i + 1) & 1]);
        return VPMC_OK;
    }));
    VPMC_TRY(finish(ctx, s, x, u, omega_out, &h));
    const double res = h.bnorm > 0 ? std::fabs(h.eta) / h.bnorm : 0.0;
    if (info) {
        info[0] = h.it;
        info[1] = res;
        info[2] = h.bnorm > 0 ? std::sqrt(h.ee) / h.bnorm : 0.0;
    }
    return res < tol || h.bnorm == 0 ? VPMC_OK : VPMC_ERR_NOT_CONVERGED;
}

}  // namespace
}  // namespace vpmc

using namespace vpmc;

extern "C" {

int vpmc_rbf_matvec(vpmc_context* ctx, int N, const float* pos, const float* x, float* y, float h_w, float Lx,
                    float Ly, int periodic, int precise) {
    if (!ctx || N < 0 || !(h_w > 0.f) || !(Lx > 0.f) || !(Ly > 0.f)) return VPMC_ERR_INVALID;
    if (N == 0) return VPMC_OK;
    if (!pos || !x || !y) return VPMC_ERR_INVALID;
    VPMC_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    Work w;
    VPMC_TRY(setup_work(ctx, SLOT_CG, N, h_w, Lx, Ly, periodic, 0, 2, &w));
    VPMC_TRY(grid_build(ctx, w.g, reinterpret_cast<const float2*>(pos), nullptr, SET_ONE_SIGNED));
    VPMC_LAUNCH(k_self_queries, work_blocks(N), 256, 0, st, w.g.cand, w.g.cstart, long(N), uint32_t(w.g.nbins),
                w.self);
    VPMC_TRY(make_items(ctx, w.g, w.g.cstart, w.it, query_chunk(4), N));
    VPMC_LAUNCH(k_gather_to_sorted<float>, work_blocks(N), 256, 0, st, x, w.g.perm, long(N), w.vec[0]);
    // FP64 pairs use W with its sigma; the FP32 form evaluates W / (2 sigma)
    VPMC_TRY(grid_set_weights_sorted(ctx, w.g, w.vec[0], precise ? 1.0 : double(w.plan.two_sigma)));
    EvalLaunch L;
    L.mode = precise ? EVAL_SPMV64 : EVAL_SPMV32;
    L.out_f64 = w.vec[1];
    VPMC_CUDA(cudaMemsetAsync(w.it.counter, 0, sizeof(uint32_t), st));
    VPMC_TRY(launch_eval(ctx, w.g, w.self, w.it, L));
    VPMC_LAUNCH(k_scatter_from_sorted, work_blocks(N), 256, 0, st, w.vec[1], w.g.perm, long(N), y);
    return vpmc_context_sync(ctx);
}

int vpmc_minres_rbf(vpmc_context* ctx, int N, const float* pos, const float* b, float* omega_out, float h_w,
                    float Lx, float Ly, int periodic, double tol, int max_iter, double* info) {
    if (!b && N > 0) return VPMC_ERR_INVALID;
    return minres_impl(ctx, N, pos, b, nullptr, omega_out, h_w, Lx, Ly, periodic, tol, max_iter, info);
}

int vpmc_minres_rbf_f64rhs(vpmc_context* ctx, int N, const float* pos, const double* b, float* omega_out, float h_w,
                           float Lx, float Ly, int periodic, double tol, int max_iter, double* info) {
    if (!b && N > 0) return VPMC_ERR_INVALID;
    return minres_impl(ctx, N, pos, nullptr, b, omega_out, h_w, Lx, Ly, periodic, tol, max_iter, info);
}

int vpmc_cg_rbf(vpmc_context* ctx, int N, const float* pos, const float* b, float* omega_out, float h_w, float Lx,
                float Ly, int periodic, double tol, int max_iter, double* info) {
    if (!b && N > 0) return VPMC_ERR_INVALID;
    return cg_impl(ctx, N, pos, b, nullptr, omega_out, h_w, Lx, Ly, periodic, tol, max_iter, info);
}

int vpmc_cg_rbf_f64rhs(vpmc_context* ctx, int N, const float* pos, const double* b, float* omega_out, float h_w,
                       float Lx, float Ly, int periodic, double tol, int max_iter, double* info) {
    if (!b && N > 0) return VPMC_ERR_INVALID;
    return cg_impl(ctx, N, pos, nullptr, b, omega_out, h_w, Lx, Ly, periodic, tol, max_iter, info);
}

}  // extern "C"
