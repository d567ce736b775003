// vpmc_eval_box.cu -- field values of densely sampled boxes by local expansions.
//
// The sum over candidates f(y) = sum w W(|y - c|) costs a square root and 8 FMA-pipe
// operations for each (sample, candidate) pair in reach.  Where hundreds of samples
// fall in a small box, most candidates are better summed once for the box: away from
// its kinks (r = h/2 and r = h) the cubic spline is 1 - 3 q + 3 q^2 - q^3 (outer) or
// 1/2 - 3 q^2 + 3 q^3 (inner) with q = |c - x| / h, and with complex c, x (units of
// h, from the box centre)
//   |c - x|^n = |c|^n sum_ab beta_a beta_b (x/c)^a conj(x/c)^b,
//   beta_a = (-1)^a binomial(n/2, a),
// so a candidate adds its terms to 21 (degree 5) moments and every sample evaluates
// one polynomial.  Candidates whose distance band across the box meets a kink, or
// that are nearer than kNear half-diagonals, are evaluated pair by pair as in k_eval.
// With boxes of at most kBoxSide h (half-diagonal rho <= 0.053) the sums are, in norm,
// more accurate than the pairwise ones, a few dozen roundings instead of 600: 9e-8 of the
// field's scale against 4e-7 for evenly spread candidates, 2.4e-7 against 4e-7 for a
// cluster of width 0.02 h.  A single value may not be: by the series' tail a candidate at
// kNear half-diagonals is off by up to 2.0e-6 of its own value at a corner of the box, one
// of the outer piece by 1.2e-7 of W(0) (the replayed series against the exact kernel;
// pair by pair 1e-7); the bound for every FP32 field value is 1e-5 of the field's scale.
// (Degree 4 is 8 % faster, but velocities next to a cluster
// were 1.3 times further from the FP64 ones than the pairwise sums, by its tail.)
// The box, not the samples in it, fixes the centre and what is expanded, so a
// sample's value does not depend on which other samples are drawn.
//
// One warp an item (a box and up to 192 of its samples): lanes are candidates while
// moments are summed and pairs collected (compacted into shared memory), and samples
// while pairs are evaluated.  512^2 particles, h_w 16, 64 + 64 samples: 16.1 ms pair by
// pair, 6.9 ms; 32 + 32 samples 8.5 and 4.2 ms; 2048^2, 64 + 64: 265 and 111 ms.  What
// bounds it is FMA issue: the pairs left (a third of the candidates, most of them in the
// bands of the two kinks) and the moments take about half of the time each.
#include <algorithm>

#include "vpmc_grid.cuh"
#include "vpmc_wide.cuh"

namespace vpmc {
namespace {

constexpr int kBoxThreads = 32;
constexpr int kPairs = kBoxChunk / 64;                 // packed sample pairs a lane
constexpr int kList = 96;                              // pairwise candidates collected before a sweep
constexpr int kRuns = 2 * (2 * 8 + 1);
constexpr float kNear = 3.f;
constexpr int kMoments = 21;

struct Run {
    uint32_t start, before;   // first candidate, candidates of the runs before
    float ox, oy;             // box centre seen through the run's image
};

template <bool K9>
__global__ void __launch_bounds__(kBoxThreads, 24) k_eval_box(EvalBoxArgs a) {
    __shared__ Run s_run[kRuns];
    __shared__ __align__(16) Cand s_list[kList];
    __shared__ float s_mom[kMoments][kBoxThreads + 1];
    __shared__ __align__(16) float s_coef[24];
    const int lane = threadIdx.x;
    const unsigned lt = (1u << lane) - 1u;
    if (a.wait_limit == 0u) {
        if (lane == 0) atomicOr(a.flags, FLAG_TIMEOUT);
        return;
    }
    uint32_t item = lane == 0 ? atomicAdd(a.counter, 1u) : 0u;
    item = __shfl_sync(0xffffffffu, item, 0);
    const uint32_t n_items = *a.n_items;
    while (item < n_items) {
        uint32_t next = lane == 0 ? atomicAdd(a.counter, 1u) : 0u;
        const Item it = a.items[item];
        const GridInst& G = a.inst[it.inst];
        const uint32_t cnt = it.qcnt & 0xffffu, box = it.qcnt >> 16;
        const uint32_t ncell = uint32_t(G.gx * G.gy), local = it.bin - uint32_t(G.bin_base);
        const uint32_t set = local / ncell, cell = local % ncell;
        const int cx = int(cell) / G.gy, cy = int(cell) % G.gy, R = a.rows, gyR = G.gy * R;
        const float sx = 1.f / G.inv_sx, sy = 1.f / G.inv_sy, ih = G.inv_hw, kap = G.B;
        // the box: a sub-cell (nb = 4), 2 x 2 sub-cells (2) or the cell (1)
        const int nb = G.nb;
        const uint2 bxy = box_coords(box, nb);
        const float inv_nb = 1.f / float(nb);
        const float bcx = (float(cx) + (float(bxy.x) + 0.5f) * inv_nb) * sx;
        const float bcy = (float(cy) + (float(bxy.y) + 0.5f) * inv_nb) * sy;
        const float hbx = 0.501f * inv_nb * sx, hby = 0.501f * inv_nb * sy;
        const float hx = hbx * ih, hy = hby * ih, rho = sqrtf(hx * hx + hy * hy);   // units of h
        const float bow = 1.25f * rho * rho;   // rho^2 / (2 (r - s)) where it matters, r - s >= 0.4

        // lane c: column c - k of the walk, its sub-rows within reach of the box
        uint32_t beg[2] = {0u, 0u}, num[2] = {0u, 0u};
        int sxi = 0, syi[2] = {0, 0};
        if (lane <= 2 * G.k) {
            const float rm = G.reach * 1.001f;
            const int ox = lane - G.k;
            int gxx = cx + ox;
            const float x0 = float(gxx) * sx, dx = fmaxf(0.f, fmaxf(x0 - (bcx + hbx), (bcx - hbx) - (x0 + sx)));
            bool col = dx < rm;
            if (G.periodic) {
                if (gxx < 0) { gxx += G.gx; sxi = -1; }
                else if (gxx >= G.gx) { gxx -= G.gx; sxi = 1; }
            } else if (gxx < 0 || gxx >= G.gx) {
                col = false;
            }
            if (col) {
                const float dy = sqrtf(fmaf(rm, rm, -dx * dx)), inv_srow = G.inv_sy * float(R);
                const int lo = floor_int(fmaf(bcy - hby - dy, inv_srow, -0.01f));
                const int hi = floor_int(fmaf(bcy + hby + dy, inv_srow, 0.01f));
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
                const uint32_t colbase = (uint32_t(G.bin_base) + set * ncell) * uint32_t(R) + uint32_t(gxx * gyR);
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (r0[h] <= r1[h]) {
                        beg[h] = a.cstart[colbase + uint32_t(r0[h])];
                        num[h] = a.cstart[colbase + uint32_t(r1[h]) + 1u] - beg[h];
                    }
            }
        }

        // this lane's samples, from the box centre (packed pairs)
        const int npw = (int(cnt) + 63) >> 6;
        f2x QX[kPairs], QY[kPairs], Q2[kPairs], ACC[kPairs];
        uint32_t qid[2 * kPairs], qfl[2 * kPairs];
        const float m2k = -2.f * kap, to_h = -0.5f * ih / kap;   // QX holds -2 kappa x; x / h = QX to_h
#pragma unroll
        for (int p = 0; p < kPairs; ++p) {
            float ax[2], ay[2];
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const uint32_t idx = uint32_t(p * 64 + s * 32 + lane);
                QRec r{bcx, bcy, kNoBin, (2u) | (2u << 3)};
                if (idx < cnt) r = a.qrec[it.qbeg + idx];
                ax[s] = r.x - bcx;
                ay[s] = r.y - bcy;
                qid[2 * p + s] = r.id;
                qfl[2 * p + s] = r.flags;
            }
            QX[p] = pk2(m2k * ax[0], m2k * ax[1]);
            QY[p] = pk2(m2k * ay[0], m2k * ay[1]);
            Q2[p] = pk2(kap * fmaf(ax[0], ax[0], ay[0] * ay[0]), kap * fmaf(ax[1], ax[1], ay[1] * ay[1]));
            ACC[p] = pk2(0.f, 0.f);
        }

        // groups of runs in one image (K9: a sample counts an image or not; otherwise
        // all runs are one group)
        unsigned left0 = __ballot_sync(0xffffffffu, num[0] > 0u), left1 = __ballot_sync(0xffffffffu, num[1] > 0u);
        const int img0 = (sxi + 1) * 3 + syi[0] + 1, img1 = (sxi + 1) * 3 + syi[1] + 1;
        while (left0 | left1) {
            int img = 4;
            unsigned g0 = left0, g1 = left1;
            if (K9) {
                img = left0 ? __shfl_sync(0xffffffffu, img0, __ffs(int(left0)) - 1)
                            : __shfl_sync(0xffffffffu, img1, __ffs(int(left1)) - 1);
                g0 &= __ballot_sync(0xffffffffu, img0 == img);
                g1 &= __ballot_sync(0xffffffffu, img1 == img);
            }
            const bool in0 = (g0 >> lane) & 1u, in1 = (g1 >> lane) & 1u;
            const uint32_t c0 = in0 ? num[0] : 0u, c1 = in1 ? num[1] : 0u;
            uint32_t incl = c0 + c1;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
            const int pos = __popc(g0 & lt) + __popc(g1 & lt), nruns = __popc(g0) + __popc(g1);
            __syncwarp();   // the runs of the previous group are read to here
            const float ox = bcx - float(sxi) * G.Lx;
            if (in0) s_run[pos] = Run{beg[0], incl - c0 - c1, ox, bcy - float(syi[0]) * G.Ly};
            if (in1) s_run[pos + (in0 ? 1 : 0)] = Run{beg[1], incl - c1, ox, bcy - float(syi[1]) * G.Ly};
            __syncwarp();

            bool use[2 * kPairs];
#pragma unroll
            for (int j = 0; j < 2 * kPairs; ++j) {
                use[j] = true;
                if (K9) {
                    const int mx = int(qfl[j] & 7u) - 2 + img / 3 - 1, my = int((qfl[j] >> 3) & 7u) - 2 + img % 3 - 1;
                    use[j] = mx >= -1 && mx <= 1 && my >= -1 && my <= 1;
                }
            }
            auto add = [&](int p, f2x v) {
                if (K9) {
                    float v0, v1;
                    up2(v, v0, v1);
                    v = pk2(use[2 * p] ? v0 : 0.f, use[2 * p + 1] ? v1 : 0.f);
                }
                ACC[p] = add2(ACC[p], v);
            };
            float m00 = 0.f, m11 = 0.f, m22 = 0.f;
            f2x m10 = pk2(0.f, 0.f), m20 = m10, m30 = m10, m40 = m10, m21 = m10, m31 = m10;
            f2x m50 = m10, m41 = m10, m32 = m10;
            int n_list = 0;
            auto sweep = [&]() {
                __syncwarp();
                f2x P[kPairs];
#pragma unroll
                for (int p = 0; p < kPairs; ++p) P[p] = pk2(0.f, 0.f);
                if (npw == 1) packed_run<1, kPairs, 4>(s_list, n_list, QX, QY, Q2, P);
                else if (npw == 2) packed_run<2, kPairs, 2>(s_list, n_list, QX, QY, Q2, P);
                else packed_run<kPairs, kPairs, 2>(s_list, n_list, QX, QY, Q2, P);
                __syncwarp();
                n_list = 0;
#pragma unroll
                for (int p = 0; p < kPairs; ++p) add(p, P[p]);   // a list at a time: short sums round less
            };
            // the candidate of flat index i (runs ascend with i in every lane), one chunk ahead
            int run = 0;
            Run rn = s_run[0];
            uint32_t run_end = nruns > 1 ? s_run[1].before : total;
            auto load = [&](uint32_t i, float& ox_, float& oy_) {
                while (i >= run_end) {
                    ++run;
                    rn = s_run[run];
                    run_end = run + 1 < nruns ? s_run[run + 1].before : total;
                }
                ox_ = rn.ox;
                oy_ = rn.oy;
                return a.cand[rn.start + (i - rn.before)];
            };
            float nox = 0.f, noy = 0.f;
            float4 nc = make_float4(0.f, 0.f, 0.f, 0.f);
            if (uint32_t(lane) < total) nc = load(uint32_t(lane), nox, noy);
#pragma unroll 1
            for (uint32_t i0 = 0; i0 < total; i0 += 32u) {
                const float4 c = nc;
                const float lx = c.x - nox, ly = c.y - noy;
                const bool valid = i0 + uint32_t(lane) < total;
                if (i0 + 32u + uint32_t(lane) < total) nc = load(i0 + 32u + uint32_t(lane), nox, noy);
                const float X = lx * ih, Y = ly * ih, r2 = fmaf(X, X, Y * Y);
                const float inv = wide::rsqrt_est(fmaxf(r2, 1e-30f)), r = r2 * inv;
                // the box's points lie between r - s and r + s + bow from the candidate, s the
                // box's half width along c and bow what the perpendicular offset adds
                const float s = fmaf(hx, fabsf(X), hy * fabsf(Y)) * inv, near = r - s, far = r + s + bow;
                const bool reach = valid && near < 1.f;
                const bool pair = reach && (far > 1.f || (near < 0.5f && far > 0.5f) || r < kNear * rho);
                const unsigned pm = __ballot_sync(0xffffffffu, pair);
                if (pair) {
                    const float c2 = kap * fmaf(lx, lx, ly * ly);
                    s_list[n_list + __popc(pm & lt)] = Cand{lx, lx, ly, ly, c.z, c.z, c2, c2};
                }
                n_list += __popc(pm);
                // only the lanes that expand: in the others 1 / c may be infinite (a candidate a
                // rounding off the box centre) or r no number (one outside an open domain by
                // 1e19 h), and a weight of 0 would make NaN of it
                if (reach && !pair) {
                    const float w = c.z;
                    const bool outer = r > 0.5f;
                    // coefficients of q, q^3 and q^2, times w
                    const float e1 = outer ? -3.f * w : 0.f, e3 = outer ? -w : 3.f * w, k2 = outer ? 3.f * w : -3.f * w;
                    const float t = 1.f - r;
                    m00 = fmaf(w, outer ? t * t * t : fmaf(-3.f * r2, t, 0.5f), m00);
                    const float A = e1 * r, B = e3 * r * r2, C = e1 * inv, D = e3 * r;
                    const float inv2 = inv * inv, E = C * inv2, F = e3 * inv;
                    const float ur = X * inv2, ui = -Y * inv2;   // 1 / c
                    const f2x U = pk2(ur, ui), IU = pk2(-ui, ur);
                    // u^m: (ar, ai) u = ar (ur, ui) + ai (-ui, ur)
                    const float vr = fmaf(ur, ur, -ui * ui), vi = 2.f * ur * ui;
                    const f2x V = pk2(vr, vi);
                    const f2x T3 = fma2(pk2(vr, vr), U, mul2(pk2(vi, vi), IU));
                    float tr, ti;
                    up2(T3, tr, ti);
                    const f2x T4 = fma2(pk2(tr, tr), U, mul2(pk2(ti, ti), IU));
                    const float f10 = fmaf(-0.5f, A, -1.5f * B) - k2 * r2;
                    const float f21 = fmaf(0.0625f, C, -0.5625f * D);
                    const float f20 = fmaf(-0.125f, A, 0.375f * B), f31 = fmaf(0.03125f, C, -0.09375f * D);
                    const float f30 = 0.0625f * (B - A), f40 = fmaf(-0.0390625f, A, 0.0234375f * B);
                    up2(T4, tr, ti);
                    const f2x T5 = fma2(pk2(tr, tr), U, mul2(pk2(ti, ti), IU));
                    const float f50 = fmaf(-0.02734375f, A, 0.01171875f * B);
                    const float f41 = fmaf(0.01953125f, C, -0.03515625f * D);
                    const float f32 = fmaf(0.0078125f, E, 0.0234375f * F);
                    m50 = fma2(pk2(f50, f50), T5, m50);
                    m41 = fma2(pk2(f41, f41), T3, m41);
                    m32 = fma2(pk2(f32, f32), U, m32);
                    m10 = fma2(pk2(f10, f10), U, m10);
                    m21 = fma2(pk2(f21, f21), U, m21);
                    m20 = fma2(pk2(f20, f20), V, m20);
                    m31 = fma2(pk2(f31, f31), V, m31);
                    m30 = fma2(pk2(f30, f30), T3, m30);
                    m40 = fma2(pk2(f40, f40), T4, m40);
                    m11 += fmaf(0.25f, C, fmaf(2.25f, D, k2));
                    m22 += fmaf(0.015625f, E, 0.140625f * F);
                }
                if (n_list > kList - 32 || (i0 + 32u >= total && n_list)) sweep();
            }

            // the lanes' moments summed, a moment a lane
            {
                const f2x* pk[9] = {&m10, &m20, &m30, &m40, &m21, &m31, &m50, &m41, &m32};
                s_mom[0][lane] = m00;
                s_mom[1][lane] = m11;
                s_mom[2][lane] = m22;
#pragma unroll
                for (int v = 0; v < 9; ++v) {
                    float re, im;
                    up2(*pk[v], re, im);
                    s_mom[3 + 2 * v][lane] = re;
                    s_mom[4 + 2 * v][lane] = im;
                }
                __syncwarp();
                if (lane < kMoments) {
                    float s0 = 0.f, s1 = 0.f;
#pragma unroll
                    for (int k = 0; k < 16; ++k) {
                        s0 += s_mom[lane][k];
                        s1 += s_mom[lane][16 + k];
                    }
                    s_coef[lane] = s0 + s1;
                }
                __syncwarp();
            }
            // f = m00 + |z|^2 (m11 + |z|^2 m22) + 2 Re[(m10 + |z|^2 (m21 + |z|^2 m32)) z
            //   + (m20 + |z|^2 m31) z^2 + (m30 + |z|^2 m41) z^3 + m40 z^4 + m50 z^5]
            const float4 k0 = *reinterpret_cast<const float4*>(&s_coef[0]), k4 = *reinterpret_cast<const float4*>(&s_coef[4]);
            const float4 k8 = *reinterpret_cast<const float4*>(&s_coef[8]), k12 = *reinterpret_cast<const float4*>(&s_coef[12]);
            const float4 k16 = *reinterpret_cast<const float4*>(&s_coef[16]);
            const float i32 = s_coef[20];
            // s_coef: m00 m11 m22 | m10 (3,4) m20 (5,6) m30 (7,8) m40 (9,10) m21 (11,12) m31 (13,14) m50 (15,16) m41 (17,18) m32 (19,20)
            const float r10 = k0.w, i10 = k4.x, r20 = k4.y, i20 = k4.z, r30 = k4.w, i30 = k8.x, r40 = k8.y, i40 = k8.z;
            const float r21 = k8.w, i21 = k12.x, r31 = k12.y, i31 = k12.z;
            const float r50 = k12.w, i50 = k16.x, r41 = k16.y, i41 = k16.z, r32 = k16.w;
            auto dup = [](float v) { return pk2(v, v); };
            const f2x TH = dup(to_h), TWO = dup(2.f);
#pragma unroll
            for (int p = 0; p < kPairs; ++p) {
                if (p >= npw) break;
                const f2x x = mul2(QX[p], TH), y = mul2(QY[p], TH), ny = mul2(y, dup(-1.f));
                const f2x x2 = mul2(x, x), y2 = mul2(y, y), q = add2(x2, y2);
                const f2x zr2 = sub2(x2, y2), xy = mul2(x, y), zi2 = add2(xy, xy);
                const f2x zr3 = fma2(zr2, x, mul2(zi2, ny)), zi3 = fma2(zr2, y, mul2(zi2, x));
                const f2x zr4 = fma2(zr2, zr2, mul2(zi2, mul2(zi2, dup(-1.f)))), zt = mul2(zr2, zi2), zi4 = add2(zt, zt);
                const f2x a1r = fma2(fma2(q, dup(r32), dup(r21)), q, dup(r10)), a1i = fma2(fma2(q, dup(i32), dup(i21)), q, dup(i10));
                const f2x a2r = fma2(q, dup(r31), dup(r20)), a2i = fma2(q, dup(i31), dup(i20));
                // Re[(ar + i ai)(zr + i zi)] = ar zr - ai zi; small terms first
                const f2x zr5 = fma2(zr4, x, mul2(zi4, ny)), zi5 = fma2(zr4, y, mul2(zi4, x));
                const f2x a3r = fma2(q, dup(r41), dup(r30)), a3i = fma2(q, dup(i41), dup(i30));
                f2x s = fma2(dup(r50), zr5, mul2(dup(-i50), zi5));
                s = fma2(dup(r40), zr4, s);
                s = fma2(dup(-i40), zi4, s);
                s = fma2(a3r, zr3, s);
                s = sub2(s, mul2(a3i, zi3));
                s = fma2(a2r, zr2, s);
                s = sub2(s, mul2(a2i, zi2));
                s = fma2(a1r, x, s);
                s = fma2(a1i, ny, s);
                const f2x e = fma2(fma2(q, dup(k0.z), dup(k0.y)), q, dup(k0.x));
                add(p, fma2(TWO, s, e));
            }
            left0 &= ~g0;
            left1 &= ~g1;
        }
#pragma unroll
        for (int p = 0; p < kPairs; ++p) {
            float v[2];
            up2(ACC[p], v[0], v[1]);
#pragma unroll
            for (int s = 0; s < 2; ++s)
                if (uint32_t(p * 64 + s * 32 + lane) < cnt) a.out[qid[2 * p + s]] = v[s] < 0.f ? 0.f : v[s];   // a NaN stays one
        }
        item = __shfl_sync(0xffffffffu, next, 0);
    }
}

}  // namespace

int launch_eval_box(vpmc_context* ctx, const EvalBoxArgs& a, bool field9) {
    int per_sm = 0;
    if (field9) {
        VPMC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_eval_box<true>, kBoxThreads, 0));
        VPMC_LAUNCH(k_eval_box<true>, ctx->sm_count * (per_sm < 1 ? 1 : per_sm), kBoxThreads, 0, ctx->stream, a);
    } else {
        VPMC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_eval_box<false>, kBoxThreads, 0));
        VPMC_LAUNCH(k_eval_box<false>, ctx->sm_count * (per_sm < 1 ? 1 : per_sm), kBoxThreads, 0, ctx->stream, a);
    }
    return VPMC_OK;
}

int box_split(long n, double samples, float Lx, float Ly, float hw, int gx, int gy) {
    const double reach = 3.14159265 * double(n) * hw * hw / (double(Lx) * Ly);
    if (reach < kBoxReach) return 0;
    const double side = std::max(double(Lx) / gx, double(Ly) / gy);
    const double per_bin = samples / (double(gx) * gy), least = kBoxSamples + kBoxFixed / reach;
    for (int nb = 1; nb <= 4; nb *= 2)
        if (side / nb <= double(kBoxSide) * hw) return per_bin >= least * nb * nb ? nb : 0;
    return 0;
}

}  // namespace vpmc
