// vpmc_direct.cu -- FP64 direct Biot-Savart sums (the accuracy oracle on the
// GPU and the "plain FP64" comparison path).
//
// Targets x sources is tiled two ways: a block owns 256 targets and one chunk
// of the sources, stages the chunk through shared memory, and writes a partial
// (u, v) per target; a second kernel adds the chunk partials in chunk order,
// so the result does not depend on scheduling.
#include <algorithm>
#include <cmath>

#include "vpmc_grid.cuh"
#include "vpmc_wide.cuh"

namespace vpmc {
namespace {

constexpr int kDT = 256;        // targets per block
constexpr int kTileSrc = 256;   // sources staged per step

template <int KERNEL>
__global__ void __launch_bounds__(kDT) k_direct(const float2* __restrict__ pos, const float* __restrict__ om,
                                                 long N, const float2* __restrict__ pts,
                                                 const int* __restrict__ tidx, long M, double param, double Lx,
                                                 double Ly, int periodic, long chunk, double2* __restrict__ part) {
    __shared__ double sx[kTileSrc], sy[kTileSrc], sw[kTileSrc];
    __shared__ int sj[kTileSrc];
    const long m = long(blockIdx.x) * kDT + threadIdx.x;
    const long c = blockIdx.y;
    const long s0 = c * chunk, s1 = min(N, s0 + chunk);
    double px = 0.0, py = 0.0;
    long self = -1;
    if (m < M) {
        if (KERNEL == VPMC_DIRECT_PLUMMER) {
            self = tidx[m];
            px = pos[self].x;
            py = pos[self].y;
        } else {
            px = pts[m].x;
            py = pts[m].y;
        }
    }
    const double e2 = param * param;
    const double inv2pi = 1.0 / (2.0 * kPiD);
    double u = 0.0, v = 0.0;
    for (long t0 = s0; t0 < s1; t0 += kTileSrc) {
        __syncthreads();
        const long j = t0 + threadIdx.x;
        if (threadIdx.x < kTileSrc) {
            if (j < s1) {
                sx[threadIdx.x] = pos[j].x;
                sy[threadIdx.x] = pos[j].y;
                sw[threadIdx.x] = om[j];
                sj[threadIdx.x] = int(j);
            } else {
                sw[threadIdx.x] = 0.0;
                sj[threadIdx.x] = -2;
            }
        }
        __syncthreads();
        const int cnt = int(min(long(kTileSrc), s1 - t0));
        for (int q = 0; q < cnt; ++q) {
            const double w = sw[q];
            if (w == 0.0) continue;
            if (KERNEL == VPMC_DIRECT_PLUMMER) {
                if (sj[q] == self) continue;
                double dx = px - sx[q], dy = py - sy[q];
                if (periodic) {
                    dx -= Lx * rint(dx / Lx);
                    dy -= Ly * rint(dy / Ly);
                }
                const double k = w * inv2pi / (dx * dx + dy * dy + e2);
                u -= dy * k;
                v += dx * k;
            } else {
                const int lo = periodic ? -1 : 0, hi = periodic ? 1 : 0;
                for (int ix = lo; ix <= hi; ++ix)
                    for (int iy = lo; iy <= hi; ++iy) {
                        const double dx = px - (sx[q] + ix * Lx);
                        const double dy = py - (sy[q] + iy * Ly);
                        const double r2 = dx * dx + dy * dy;
                        if (r2 == 0.0) continue;
                        double k = w * inv2pi / r2;
                        if (r2 < param * param) k *= spline_mass_d(sqrt(r2) / param);
                        u -= dy * k;
                        v += dx * k;
                    }
            }
        }
    }
    if (m < M) part[c * M + m] = make_double2(u, v);
}

// FP32 tiles: the deterministic "P" particle method of the reference
// (biot_savart_naive_kernel, src/cuda/naive_biot_savart.cu:15-40, is FP32).
__device__ __forceinline__ float spline_mass_f(float q) {
    if (q >= 1.f) return 1.f;
    const float c = 80.f / 7.f, q2 = q * q;
    if (q <= 0.5f) return c * q2 * fmaf(q2, fmaf(1.2f, q, -1.5f), 0.5f);
    const float g = q2 * fmaf(q2, fmaf(-0.4f, q, 1.5f), fmaf(-2.f, q, 1.f));
    return c * (0.06875f + g - 0.08125f);
}

template <int KERNEL>
__global__ void __launch_bounds__(kDT) k_direct_f32(const float2* __restrict__ pos, const float* __restrict__ om,
                                                     long N, const float2* __restrict__ pts,
                                                     const int* __restrict__ tidx, long M, float param, float Lx,
                                                     float Ly, int periodic, long chunk, float2* __restrict__ part) {
    __shared__ float2 sp[kTileSrc];
    __shared__ float sw[kTileSrc];
    __shared__ int sj[kTileSrc];
    const long m = long(blockIdx.x) * kDT + threadIdx.x;
    const long c = blockIdx.y;
    const long s0 = c * chunk, s1 = min(N, s0 + chunk);
    float2 x = make_float2(0.f, 0.f);
    long self = -1;
    if (m < M) {
        if (KERNEL == VPMC_DIRECT_PLUMMER) { self = tidx[m]; x = pos[self]; }
        else x = pts[m];
    }
    const float e2 = param * param, inv2pi = 1.f / (2.f * kPiF), ih = 1.f / param;
    float u = 0.f, v = 0.f;
    for (long t0 = s0; t0 < s1; t0 += kTileSrc) {
        __syncthreads();
        const long j = t0 + threadIdx.x;
        if (threadIdx.x < kTileSrc) {
            sp[threadIdx.x] = j < s1 ? pos[j] : make_float2(0.f, 0.f);
            sw[threadIdx.x] = j < s1 ? om[j] : 0.f;
            sj[threadIdx.x] = j < s1 ? int(j) : -2;
        }
        __syncthreads();
        const int cnt = int(min(long(kTileSrc), s1 - t0));
        for (int q = 0; q < cnt; ++q) {
            const float w = sw[q];
            if (KERNEL == VPMC_DIRECT_PLUMMER) {
                if (sj[q] == self) continue;
                float dx = x.x - sp[q].x, dy = x.y - sp[q].y;
                if (periodic) {   // wrap_min_image (include/monte_carlo_bs.cuh:140-143)
                    dx -= rintf(dx / Lx) * Lx;
                    dy -= rintf(dy / Ly) * Ly;
                }
                const float k = w * inv2pi / (dx * dx + dy * dy + e2);
                u -= dy * k;
                v += dx * k;
            } else {
                const int lo = periodic ? -1 : 0, hi = periodic ? 1 : 0;
                for (int ix = lo; ix <= hi; ++ix)
                    for (int iy = lo; iy <= hi; ++iy) {
                        const float dx = x.x - (sp[q].x + ix * Lx), dy = x.y - (sp[q].y + iy * Ly);
                        const float r2 = dx * dx + dy * dy;
                        if (r2 == 0.f) continue;
                        float k = w * inv2pi / r2;
                        if (r2 < e2) k *= spline_mass_f(sqrtf(r2) * ih);
                        u -= dy * k;
                        v += dx * k;
                    }
            }
        }
    }
    if (m < M) part[c * M + m] = make_float2(u, v);
}

// The mollified FP64 sum on a periodic domain.  The FP64 pipe bounds it (2
// lanes a clock and SM), so the kernel is written for few FP64 instructions:
// the three images of a row (same dy) share one reciprocal,
//   sum 1/r2 = (ab + bc + ca) / (abc),  sum dx/r2 = (dx_a bc + dx_b ac + dx_c ab) / (abc),
// whose terms are all positive products (no cancellation that the separate
// quotients do not have), the reciprocal is the hardware's 20-bit estimate with
// one third-order step, y (1 + e + e^2) with e = 1 - d y (Householder's iteration
// for 1 / d; 2^28 divisors over the exponent range: an ulp beside 1.0 / d for 3 in
// 10,000, |1 - d y| at most 1.115e-16), and 1/(2 pi)
// multiplies the chunk's sum.  67 FP64 instructions a source and target against
// about 200 for nine quotients: 4,096 targets x 262,144 sources, 311.2 -> 141.6 ms.
// A row with an image inside the mollifier (or at r = 0, or with a non-finite
// distance or strength) takes the quotients one by one.
__device__ __forceinline__ double rcp_f64(double d) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = fma(-d, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

__global__ void __launch_bounds__(kDT) k_direct_rows(const float2* __restrict__ pos, const float* __restrict__ om,
                                                      long N, const float2* __restrict__ pts, long M, double param,
                                                      double Lx, double Ly, long chunk, double2* __restrict__ part) {
    __shared__ double sx[kTileSrc][3], sy[kTileSrc][3], sw[kTileSrc];
    const long m = long(blockIdx.x) * kDT + threadIdx.x;
    const long c = blockIdx.y;
    const long s0 = c * chunk, s1 = min(N, s0 + chunk);
    const double px = m < M ? double(pts[m].x) : 0.0, py = m < M ? double(pts[m].y) : 0.0;
    const double p2 = param * param;
    const int near_hi = __double2hiint(p2);
    double u = 0.0, v = 0.0;
    for (long t0 = s0; t0 < s1; t0 += kTileSrc) {
        __syncthreads();
        const long j = t0 + threadIdx.x;
        if (j < s1) {
            const double x = pos[j].x, y = pos[j].y;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                sx[threadIdx.x][i] = x + (i - 1) * Lx;
                sy[threadIdx.x][i] = y + (i - 1) * Ly;
            }
            sw[threadIdx.x] = om[j];
        }
        __syncthreads();
        const int cnt = int(min(long(kTileSrc), s1 - t0));
        for (int q = 0; q < cnt; ++q) {
            const double w = sw[q];
            if (w == 0.0) continue;
            const bool wild = (__double2hiint(w) & 0x7ff00000) == 0x7ff00000;
            double dx[3], X[3], su = 0.0, sv = 0.0;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                dx[i] = px - sx[q][i];
                X[i] = dx[i] * dx[i];
            }
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                const double dy = py - sy[q][r];
                const double a = fma(dy, dy, X[0]), b = fma(dy, dy, X[1]), cc = fma(dy, dy, X[2]);
                const double ab = a * b, bc = b * cc, ac = a * cc, den = ab * cc;
                // the high words order as the (non-negative) values do; NaN and infinity are the largest
                const int lo = min(__double2hiint(a), min(__double2hiint(b), __double2hiint(cc)));
                const unsigned dh = unsigned(__double2hiint(den)) - 0x00200000u;   // outside [2^-1020, inf) or NaN
                if (wild || lo <= near_hi || dh >= 0x7ff00000u - 0x00200000u) {
                    const double r2s[3] = {a, b, cc};
                    for (int i = 0; i < 3; ++i) {
                        const double r2 = r2s[i];
                        if (r2 == 0.0) continue;
                        double k = w / r2;
                        if (r2 < p2) k *= spline_mass_d(sqrt(r2) / param);
                        u -= dy * k;
                        v += dx[i] * k;
                    }
                } else {
                    const double inv = rcp_f64(den);
                    su = fma(dy, (ab + bc + ac) * inv, su);
                    sv = fma(fma(dx[0], bc, fma(dx[1], ac, dx[2] * ab)), inv, sv);
                }
            }
            if (!wild) {
                u = fma(-w, su, u);
                v = fma(w, sv, v);
            }
        }
    }
    const double inv2pi = 1.0 / (2.0 * kPiD);
    if (m < M) part[c * M + m] = make_double2(u * inv2pi, v * inv2pi);
}

// The same sum in three-float arithmetic (vpmc_wide.cuh) on the FP32 pipe, which
// has 64 times the FP64 pipe's lanes: about 1,000 FP32 instructions a source and
// target (nine reciprocals and the row and column sums of the reciprocals, the
// differences once a row and column), each term to 2^-65, a tile's sum added in
// FP64.  4,096 targets x 262,144 sources: 141.6 -> 42.4 ms (311.2 at first); the error
// against a 64-bit restatement went from 1.5e-15 to 4e-16, that of the restatement.
// Images inside the mollifier (or at a distance the floats' parts cannot hold) are
// noted per thread and added in FP64 after the tile, all lanes at once: 9% of the
// (warp, source) pairs have one.  A tile with a non-finite strength, or strengths
// whose range exceeds 1e15, is summed in FP64 throughout.
constexpr int kWideNotes = 12;

__device__ __forceinline__ void mollified_pair(double dx, double dy, double w, double param, double& u, double& v) {
    const double r2 = dx * dx + dy * dy;
    if (r2 == 0.0) return;
    double k = w / r2;
    if (r2 < param * param) k *= spline_mass_d(sqrt(r2) / param);
    u -= dy * k;
    v += dx * k;
}

__global__ void __launch_bounds__(kDT, 2) k_direct_wide(const float2* __restrict__ pos, const float* __restrict__ om,
                                                         long N, const float2* __restrict__ pts, long M, double param,
                                                         float Lx, float Ly, float near2, long chunk,
                                                         double2* __restrict__ part) {
    __shared__ float4 s_x[kTileSrc], s_xl[kTileSrc], s_y[kTileSrc], s_yl[kTileSrc];   // images -1, 0, 1; strength in s_x.w
    __shared__ uint16_t s_note[kWideNotes][kDT];
    __shared__ float s_most[kDT / 32], s_least[kDT / 32];
    const int tid = threadIdx.x;
    const long m = long(blockIdx.x) * kDT + tid, c = blockIdx.y;
    const long s0 = c * chunk, s1 = min(N, s0 + chunk);
    const float px = m < M ? pts[m].x : 0.f, py = m < M ? pts[m].y : 0.f;
    double u = 0.0, v = 0.0;
    for (long t0 = s0; t0 < s1; t0 += kTileSrc) {
        const int cnt = int(min(long(kTileSrc), s1 - t0));
        float most = 0.f, least = INFINITY;
        bool finite = true;
        if (tid < cnt) {
            const float2 p = pos[t0 + tid];
            const float w = om[t0 + tid], a = fabsf(w);
            float4 x, xl, y, yl;
            wide::two_sum(p.x, -Lx, x.x, xl.x);
            wide::two_sum(p.x, Lx, x.z, xl.z);
            wide::two_sum(p.y, -Ly, y.x, yl.x);
            wide::two_sum(p.y, Ly, y.z, yl.z);
            x.y = p.x;
            y.y = p.y;
            xl.y = yl.y = xl.w = y.w = yl.w = 0.f;
            x.w = w;
            s_x[tid] = x;
            s_xl[tid] = xl;
            s_y[tid] = y;
            s_yl[tid] = yl;
            finite = a <= 3.0e38f;
            most = a;
            if (a > 0.f) least = a;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
            least = fminf(least, __shfl_xor_sync(0xffffffffu, least, o));
        }
        if ((tid & 31) == 0) {
            s_most[tid >> 5] = most;
            s_least[tid >> 5] = least;
        }
        finite = __syncthreads_and(finite);
#pragma unroll
        for (int k = 0; k < kDT / 32; ++k) {
            most = fmaxf(most, s_most[k]);
            least = fminf(least, s_least[k]);
        }
        // the strengths times a power of two: the largest is about 1
        const int ex = min(max(254 - int(__float_as_uint(most) >> 23), 1), 253);
        const float scale = __uint_as_float(uint32_t(ex) << 23);
        const bool fits = finite && (most == 0.f || least * scale >= 1e-15f);
        if (fits) {
            wide::W3 su{0.f, 0.f, 0.f}, sv{0.f, 0.f, 0.f};
            int notes = 0;
#pragma unroll 1
            for (int q = 0; q < cnt; ++q) {
                const float4 x = s_x[q], xl = s_xl[q], y = s_y[q], yl = s_yl[q];
                const float w = x.w * scale;
                if (w == 0.f) continue;
                wide::W3 X[3], C[3], U;
                float dh[3], dl[3];
                const float xs[3] = {x.x, x.y, x.z}, xls[3] = {xl.x, xl.y, xl.z};
                const float ys[3] = {y.x, y.y, y.z}, yls[3] = {yl.x, yl.y, yl.z};
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    float a, e;
                    wide::two_sum(px, -xs[i], a, e);
                    wide::fast_two_sum(a, wide::sub(e, xls[i]), dh[i], dl[i]);
                    X[i] = wide::sqr3(wide::W3{dh[i], dl[i], 0.f});
                }
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    float a, e, eh, el;
                    wide::two_sum(py, -ys[j], a, e);
                    wide::fast_two_sum(a, wide::sub(e, yls[j]), eh, el);
                    const wide::W3 Y = wide::sqr3(wide::W3{eh, el, 0.f});
                    wide::W3 S;
#pragma unroll
                    for (int i = 0; i < 3; ++i) {
                        const wide::W3 r2 = wide::add3(X[i], Y);
                        wide::W3 k = wide::rcp3(r2);
                        if (!(r2.a > near2 && r2.a < 1e30f)) {
                            k = wide::W3{0.f, 0.f, 0.f};
                            if (notes < kWideNotes) s_note[notes][tid] = uint16_t(q * 16 + j * 4 + i);
                            else mollified_pair(double(px) - (double(xs[i]) + double(xls[i])),
                                                double(py) - (double(ys[j]) + double(yls[j])), double(x.w), param, u, v);
                            ++notes;
                        }
                        S = i ? wide::add3(S, k) : k;
                        C[i] = j ? wide::add3(C[i], k) : k;
                    }
                    const wide::W3 p = wide::mul2(eh, el, S);
                    U = j ? wide::add3(U, p) : p;
                }
                const wide::W3 V = wide::add3(wide::add3(wide::mul2(dh[0], dl[0], C[0]), wide::mul2(dh[1], dl[1], C[1])),
                                              wide::mul2(dh[2], dl[2], C[2]));
                su = wide::norm3(wide::add3(su, wide::mul1(-w, U)));
                sv = wide::norm3(wide::add3(sv, wide::mul1(w, V)));
            }
            const double unit = 1.0 / double(scale);
            u += ((double(su.a) + double(su.b)) + double(su.c)) * unit;
            v += ((double(sv.a) + double(sv.b)) + double(sv.c)) * unit;
            for (int n = 0; n < min(notes, kWideNotes); ++n) {
                const int id = s_note[n][tid], q = id >> 4, j = (id >> 2) & 3, i = id & 3;
                const float* xs = &s_x[q].x;
                const float* ys = &s_y[q].x;
                mollified_pair(double(px) - (double(xs[i]) + double((&s_xl[q].x)[i])),
                               double(py) - (double(ys[j]) + double((&s_yl[q].x)[j])), double(s_x[q].w), param, u, v);
            }
        } else {
            for (int q = 0; q < cnt; ++q) {
                const float* xs = &s_x[q].x;
                const float* ys = &s_y[q].x;
                if (s_x[q].w == 0.f) continue;
                for (int i = 0; i < 3; ++i)
                    for (int j = 0; j < 3; ++j)
                        mollified_pair(double(px) - (double(xs[i]) + double((&s_xl[q].x)[i])),
                                       double(py) - (double(ys[j]) + double((&s_yl[q].x)[j])), double(s_x[q].w), param, u,
                                       v);
            }
        }
        __syncthreads();   // the tile and s_most are read to here
    }
    const double inv2pi = 1.0 / (2.0 * kPiD);
    if (m < M) part[c * M + m] = make_double2(u * inv2pi, v * inv2pi);
}

// The Plummer "P" method in FP32, four targets a thread in two packed pairs.
// The FP32 pipe bounds it: 13 packed instructions and two reciprocals a source
// and pair of targets (differences 2, minimum image 6, r2 2, strength 1, sums
// 2), sources broadcast from shared memory with their operands duplicated.  The
// minimum image is rint(dx / L) by a multiplication with 1/L and the add of 1.5
// 2^23; for a period that is a power of two (kExact) the product is the quotient,
// otherwise a pair within 1e-4 of the tie takes the IEEE quotient, so the image
// chosen is always the quotient's.  Each thread adds a tile's sum at a time, so
// its rounding error grows with the tile (64 sources) and the number of tiles,
// not with the chunk (40,000 particles: 4.8e-6 of the FP64 sum, before 4.9e-6;
// the rounding of the FP32 differences is most of it, with the estimate's reciprocal,
// an ulp off at most, as with the IEEE quotient).
// 40,000 targets x 40,000 sources: 3,217 -> 697 us, 29.8 TFLOP/s at 13 flop a pair.
// A tile with a source (or a block with a target) many periods away (2^20, or
// 256 where the product with 1/L is rounded), without periods 2^61 away (beyond,
// r2 may pass 2^126, whose reciprocal the estimate flushes to 0), or with a
// strength that could overflow against e2 takes the general arithmetic.
constexpr int kPT = 128;          // threads
constexpr int kPTargets = 4;      // targets a thread
constexpr int kPTile = 64;        // sources a tile

struct __align__(16) PSrc {
    float x, x2, y, y2, w, w2, pad, pad2;
};

__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// dx - rint(dx / L) L of a packed pair
template <bool kExact>
__device__ __forceinline__ f2x min_image2(f2x d, f2x iL, f2x nL, float L) {
    const float kMagic = 12582912.f;   // 1.5 2^23: the add rounds to an integer
    const f2x M = pk2(kMagic, kMagic), nM = pk2(-kMagic, -kMagic);
    f2x k = add2(fma2(d, iL, M), nM);
    if constexpr (!kExact) {
        float da, db, ka, kb, fa, fb;
        up2(d, da, db);
        up2(k, ka, kb);
        up2(fma2(d, iL, mul2(k, pk2(-1.f, -1.f))), fa, fb);
        if (fabsf(fa) > 0.4999f || fabsf(fb) > 0.4999f) {
            ka = rintf(da / L);
            kb = rintf(db / L);
            k = pk2(ka, kb);
        }
    }
    return fma2(k, nL, d);
}

template <bool kPeriodic, bool kExact>
__global__ void __launch_bounds__(kPT) k_plummer_f32(const float2* __restrict__ pos, const float* __restrict__ om,
                                                      long N, const int* __restrict__ tidx, long M, float param,
                                                      float Lx, float Ly, long chunk, float2* __restrict__ part) {
    __shared__ PSrc src[kPTile];
    const long c = blockIdx.y;
    const long s0 = c * chunk, s1 = min(N, s0 + chunk);
    const long m0 = long(blockIdx.x) * (kPT * kPTargets) + threadIdx.x;
    const float e2 = param * param, inv2pi = 1.f / (2.f * kPiF), iLx = 1.f / Lx, iLy = 1.f / Ly;
    constexpr float kFar = !kPeriodic ? 0x1p61f : kExact ? 1048576.f : 256.f;   // periods, or lengths without them
    const float ux = kPeriodic ? iLx : 1.f, uy = kPeriodic ? iLy : 1.f;
    const float wmax = 3.0e38f * fminf(e2, 1.f);
    float2 x[kPTargets];
    int self[kPTargets];
    bool far = false;
#pragma unroll
    for (int j = 0; j < kPTargets; ++j) {
        const long m = m0 + long(j) * kPT;
        self[j] = m < M ? tidx[m] : -1;
        x[j] = m < M ? pos[self[j]] : make_float2(0.f, 0.f);
        far |= !(fabsf(x[j].x) * ux < kFar && fabsf(x[j].y) * uy < kFar);
    }
    f2x X[2], Y[2], U[2], V[2];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        X[p] = pk2(x[2 * p].x, x[2 * p + 1].x);
        Y[p] = pk2(x[2 * p].y, x[2 * p + 1].y);
        U[p] = V[p] = pk2(0.f, 0.f);
    }
    const f2x IX = pk2(iLx, iLx), IY = pk2(iLy, iLy), NX = pk2(-Lx, -Lx), NY = pk2(-Ly, -Ly), E2 = pk2(e2, e2);
    const f2x ZERO = pk2(0.f, 0.f);
    for (long t0 = s0; t0 < s1; t0 += kPTile) {
        const int cnt = int(min(long(kPTile), s1 - t0));
        bool general = far;
        if (threadIdx.x < cnt) {
            const float2 p = pos[t0 + threadIdx.x];
            const float w = om[t0 + threadIdx.x] * inv2pi;
            src[threadIdx.x] = PSrc{-p.x, -p.x, -p.y, -p.y, w, w, 0.f, 0.f};
            general |= !(fabsf(w) <= wmax);
            general |= !(fabsf(p.x) * ux < kFar && fabsf(p.y) * uy < kFar);
        }
        f2x tu[2] = {ZERO, ZERO}, tv[2] = {ZERO, ZERO};
        if (!__syncthreads_or(general)) {
#pragma unroll 4
            for (int q = 0; q < cnt; ++q) {
                const ulonglong2 P = *reinterpret_cast<const ulonglong2*>(&src[q].x);
                const f2x W = *reinterpret_cast<const f2x*>(&src[q].w);
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    f2x dx = add2(X[p], P.x), dy = add2(Y[p], P.y);
                    if (kPeriodic) {
                        dx = min_image2<kExact>(dx, IX, NX, Lx);
                        dy = min_image2<kExact>(dy, IY, NY, Ly);
                    }
                    // the target itself adds exact zeros (dx = dy = 0, r2 + e2 > 0)
                    float da, db;
                    up2(fma2(dx, dx, fma2(dy, dy, E2)), da, db);
                    const f2x K = mul2(W, pk2(rcp_approx(da), rcp_approx(db)));
                    tu[p] = fma2(dy, K, tu[p]);
                    tv[p] = fma2(dx, K, tv[p]);
                }
            }
        } else {
            for (int q = 0; q < cnt; ++q) {
                float k2[2][2][2];
#pragma unroll
                for (int j = 0; j < kPTargets; ++j) {
                    float dx = x[j].x + src[q].x, dy = x[j].y + src[q].y;
                    if (kPeriodic) {
                        dx -= rintf(dx / Lx) * Lx;
                        dy -= rintf(dy / Ly) * Ly;
                    }
                    const float k = src[q].w / (dx * dx + dy * dy + e2);
                    const bool me = int(t0) + q == self[j];
                    k2[j >> 1][j & 1][0] = me ? 0.f : dy * k;
                    k2[j >> 1][j & 1][1] = me ? 0.f : dx * k;
                }
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    tu[p] = add2(tu[p], pk2(k2[p][0][0], k2[p][1][0]));
                    tv[p] = add2(tv[p], pk2(k2[p][0][1], k2[p][1][1]));
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            U[p] = add2(U[p], tu[p]);
            V[p] = add2(V[p], tv[p]);
        }
    }
#pragma unroll
    for (int j = 0; j < kPTargets; ++j) {
        const long m = m0 + long(j) * kPT;
        float ua, ub, va, vb;
        up2(U[j >> 1], ua, ub);
        up2(V[j >> 1], va, vb);
        if (m < M) part[c * M + m] = make_float2(-((j & 1) ? ub : ua), (j & 1) ? vb : va);
    }
}

__global__ void k_direct_reduce_f32(const float2* __restrict__ part, long M, int nchunk, float* __restrict__ out) {
    for (long m = long(blockIdx.x) * blockDim.x + threadIdx.x; m < M; m += long(gridDim.x) * blockDim.x) {
        float u = 0.f, v = 0.f;
        for (int c = 0; c < nchunk; ++c) {
            const float2 p = part[long(c) * M + m];
            u += p.x;
            v += p.y;
        }
        out[2 * m] = u;
        out[2 * m + 1] = v;
    }
}

__global__ void k_direct_reduce(const double2* __restrict__ part, long M, int nchunk, double* __restrict__ out) {
    for (long m = long(blockIdx.x) * blockDim.x + threadIdx.x; m < M; m += long(gridDim.x) * blockDim.x) {
        double u = 0.0, v = 0.0;
        for (int c = 0; c < nchunk; ++c) {
            const double2 p = part[long(c) * M + m];
            u += p.x;
            v += p.y;
        }
        out[2 * m] = u;
        out[2 * m + 1] = v;
    }
}

}  // namespace
}  // namespace vpmc

using namespace vpmc;

extern "C" int vpmc_direct_velocity_f64(vpmc_context* ctx, int kernel, int N, const float* pos, const float* omega,
                                        int M, const float* pts, const int* tidx, double param, double Lx, double Ly,
                                        int periodic, double* out_uv) {
    if (!ctx || N < 0 || M < 0 || !(Lx > 0) || !(Ly > 0)) return VPMC_ERR_INVALID;
    if (kernel != VPMC_DIRECT_MOLLIFIED && kernel != VPMC_DIRECT_PLUMMER) return VPMC_ERR_INVALID;
    if (M == 0) return VPMC_OK;
    if (!out_uv || (N > 0 && (!pos || !omega))) return VPMC_ERR_INVALID;
    if (kernel == VPMC_DIRECT_PLUMMER ? !tidx : !pts) return VPMC_ERR_INVALID;
    if (kernel == VPMC_DIRECT_MOLLIFIED && !(param > 0)) return VPMC_ERR_INVALID;
    VPMC_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    const long tblocks = (long(M) + kDT - 1) / kDT;
    // three-float arithmetic: periods that are floats of ordinary size; images within
    // the core, or closer than 1e-9 periods, are added in FP64
    const double Lmin = std::min(Lx, Ly), Lmax = std::max(Lx, Ly);
    const bool wide = double(float(Lx)) == Lx && double(float(Ly)) == Ly && Lmin >= 1e-5 && Lmax <= 1e5 &&
                      Lmax <= 1e3 * Lmin && param <= Lmax;
    const float near2 = float(std::max(param * param, 1e-18 * Lmax * Lmax) * (1.0 + 1e-6));
    // enough blocks to fill the GPU several times over
    long nchunk = (8L * ctx->sm_count + tblocks - 1) / tblocks;
    if (nchunk < 1) nchunk = 1;
    if (nchunk > 4096) nchunk = 4096;
    long chunk = (long(N) + nchunk - 1) / nchunk;
    if (chunk < kTileSrc) chunk = kTileSrc;
    nchunk = N > 0 ? (long(N) + chunk - 1) / chunk : 1;
    char* base = nullptr;
    VPMC_TRY(scratch(ctx, SLOT_DIRECT, sizeof(double2) * size_t(nchunk) * size_t(M) + 256, &base));
    double2* part = reinterpret_cast<double2*>(base);
    if (N == 0) {
        VPMC_CUDA(cudaMemsetAsync(part, 0, sizeof(double2) * size_t(M), st));
    } else {
        const dim3 grid{static_cast<unsigned>(tblocks), static_cast<unsigned>(nchunk), 1u};
        if (kernel == VPMC_DIRECT_PLUMMER)
            VPMC_LAUNCH(k_direct<VPMC_DIRECT_PLUMMER>, grid, kDT, 0, st, reinterpret_cast<const float2*>(pos), omega,
                        long(N), nullptr, tidx, long(M), param, Lx, Ly, periodic, chunk, part);
        else if (periodic && wide)
            VPMC_LAUNCH(k_direct_wide, grid, kDT, 0, st, reinterpret_cast<const float2*>(pos), omega, long(N),
                        reinterpret_cast<const float2*>(pts), long(M), param, float(Lx), float(Ly), near2, chunk, part);
        else if (periodic)
            VPMC_LAUNCH(k_direct_rows, grid, kDT, 0, st, reinterpret_cast<const float2*>(pos), omega, long(N),
                        reinterpret_cast<const float2*>(pts), long(M), param, Lx, Ly, chunk, part);
        else
            VPMC_LAUNCH(k_direct<VPMC_DIRECT_MOLLIFIED>, grid, kDT, 0, st, reinterpret_cast<const float2*>(pos),
                        omega, long(N), reinterpret_cast<const float2*>(pts), nullptr, long(M), param, Lx, Ly,
                        periodic, chunk, part);
    }
    VPMC_LAUNCH(k_direct_reduce, unsigned((M + 255) / 256), 256, 0, st, part, long(M), int(nchunk), out_uv);
    return vpmc_context_sync(ctx);
}

extern "C" int vpmc_direct_velocity_f32(vpmc_context* ctx, int kernel, int N, const float* pos, const float* omega,
                                        int M, const float* pts, const int* tidx, float param, float Lx, float Ly,
                                        int periodic, float* out_uv) {
    if (!ctx || N < 0 || M < 0 || !(Lx > 0.f) || !(Ly > 0.f)) return VPMC_ERR_INVALID;
    if (kernel != VPMC_DIRECT_MOLLIFIED && kernel != VPMC_DIRECT_PLUMMER) return VPMC_ERR_INVALID;
    if (M == 0) return VPMC_OK;
    if (!out_uv || (N > 0 && (!pos || !omega))) return VPMC_ERR_INVALID;
    if (kernel == VPMC_DIRECT_PLUMMER ? !tidx : !pts) return VPMC_ERR_INVALID;
    if (kernel == VPMC_DIRECT_MOLLIFIED && !(param > 0.f)) return VPMC_ERR_INVALID;
    VPMC_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    // the packed Plummer kernel wants r2 + e2 in the reciprocal's normal range (e2
    // bounds it below, the period above); a smaller or huge core and a huge period
    // keep the IEEE quotients
    const float e2 = param * param;
    const bool packed = kernel == VPMC_DIRECT_PLUMMER && e2 >= 1e-30f && e2 <= 1e30f &&
                        !(periodic && std::max(Lx, Ly) > 0x1p61f);
    const long per_block = packed ? long(kPT) * kPTargets : long(kDT);
    const long tile = packed ? kPTile : kTileSrc;
    const long tblocks = (long(M) + per_block - 1) / per_block;
    // packed: 16 blocks of 128 threads fill an SM
    long nchunk = ((packed ? 16L : 8L) * ctx->sm_count + tblocks - 1) / tblocks;
    if (nchunk < 1) nchunk = 1;
    if (nchunk > 4096) nchunk = 4096;
    long chunk = (long(N) + nchunk - 1) / nchunk;
    if (packed) chunk = (chunk + tile - 1) / tile * tile;
    // (few targets: the chunks' partials are added one after the other, 55 ns each, so a
    // chunk is four tiles at least: 50,000 sources, 100 targets, no period, 102 us a call
    // with 782 chunks, 63 with 196, 83 before the tiles were packed; 600 targets 121, 74
    // and 100)
    const long least = packed && tblocks <= 2 ? 4 * tile : tile;
    if (chunk < least) chunk = least;
    nchunk = N > 0 ? (long(N) + chunk - 1) / chunk : 1;
    char* base = nullptr;
    VPMC_TRY(scratch(ctx, SLOT_DIRECT, sizeof(float2) * size_t(nchunk) * size_t(M) + 256, &base));
    float2* part = reinterpret_cast<float2*>(base);
    if (N == 0) {
        VPMC_CUDA(cudaMemsetAsync(part, 0, sizeof(float2) * size_t(M), st));
    } else {
        const dim3 grid{static_cast<unsigned>(tblocks), static_cast<unsigned>(nchunk), 1u};
        if (packed) {
            const auto pow2 = [](float L) {   // 1/L and dx (1/L) are exact: the product is the quotient
                int e;
                return std::frexp(L, &e) == 0.5f && e > -100 && e < 100;
            };
            const float2* p2 = reinterpret_cast<const float2*>(pos);
            if (!periodic)
                VPMC_LAUNCH((k_plummer_f32<false, true>), grid, kPT, 0, st, p2, omega, long(N), tidx, long(M), param,
                            Lx, Ly, chunk, part);
            else if (pow2(Lx) && pow2(Ly))
                VPMC_LAUNCH((k_plummer_f32<true, true>), grid, kPT, 0, st, p2, omega, long(N), tidx, long(M), param,
                            Lx, Ly, chunk, part);
            else
                VPMC_LAUNCH((k_plummer_f32<true, false>), grid, kPT, 0, st, p2, omega, long(N), tidx, long(M), param,
                            Lx, Ly, chunk, part);
        } else if (kernel == VPMC_DIRECT_PLUMMER)
            VPMC_LAUNCH(k_direct_f32<VPMC_DIRECT_PLUMMER>, grid, kDT, 0, st, reinterpret_cast<const float2*>(pos),
                        omega, long(N), nullptr, tidx, long(M), param, Lx, Ly, periodic, chunk, part);
        else
            VPMC_LAUNCH(k_direct_f32<VPMC_DIRECT_MOLLIFIED>, grid, kDT, 0, st, reinterpret_cast<const float2*>(pos),
                        omega, long(N), reinterpret_cast<const float2*>(pts), nullptr, long(M), param, Lx, Ly,
                        periodic, chunk, part);
    }
    VPMC_LAUNCH(k_direct_reduce_f32, unsigned((M + 255) / 256), 256, 0, st, part, long(M), int(nchunk), out_uv);
    return vpmc_context_sync(ctx);
}
