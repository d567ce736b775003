// vpmc_wide.cuh -- FP64-grade kernel sums on the FP32 pipe.
//
// sm_103a has 2 FP64 lanes a clock and SM against 128 FP32 lanes, so an FP64
// instruction costs as much as 64 FP32 ones.  A number is held here as an
// unevaluated sum of three floats (about 70 bits) and computed with error-free
// sums and products (Knuth's TwoSum, Dekker's FastTwoSum, the FMA product error:
// Ogita, Rump & Oishi, SIAM J. Sci. Comput. 26, 2005).  The terms are closer to
// the exact ones than FP64 arithmetic's (whose own roundings are 2^-53 each).
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define VPMC_WIDE_FN __device__ __forceinline__
#else
#define VPMC_WIDE_FN inline
#endif

namespace vpmc {
namespace wide {

// IEEE single operations that no compiler contracts or reorders.
#ifdef __CUDA_ARCH__
VPMC_WIDE_FN float add(float a, float b) { return __fadd_rn(a, b); }
VPMC_WIDE_FN float sub(float a, float b) { return __fsub_rn(a, b); }
VPMC_WIDE_FN float mul(float a, float b) { return __fmul_rn(a, b); }
VPMC_WIDE_FN float fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
VPMC_WIDE_FN float rsqrt_est(float a) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}
VPMC_WIDE_FN float rcp_est(float a) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}
#else
VPMC_WIDE_FN float add(float a, float b) { return a + b; }
VPMC_WIDE_FN float sub(float a, float b) { return a - b; }
VPMC_WIDE_FN float mul(float a, float b) { return a * b; }
VPMC_WIDE_FN float fma(float a, float b, float c) { return std::fmaf(a, b, c); }
VPMC_WIDE_FN float rsqrt_est(float a) { return 1.f / std::sqrt(a); }
VPMC_WIDE_FN float rcp_est(float a) { return 1.f / a; }
#endif

VPMC_WIDE_FN void two_sum(float a, float b, float& s, float& e) {
    s = add(a, b);
    const float t = sub(s, a);
    e = add(sub(a, sub(s, t)), sub(b, t));
}
VPMC_WIDE_FN void fast_two_sum(float a, float b, float& s, float& e) {   // |a| >= |b| (or a = 0)
    s = add(a, b);
    e = sub(b, sub(s, a));
}
VPMC_WIDE_FN void two_prod(float a, float b, float& p, float& e) {
    p = mul(a, b);
    e = fma(a, b, -p);
}

struct W3 {
    float a, b, c;   // a + b + c, |b| <= ulp(a), |c| ~ ulp(b)
};

// x y of two wide numbers (unnormalised: the parts overlap by a bit or two).
VPMC_WIDE_FN W3 mul3(const W3& x, const W3& y) {
    float p, e, q, eq, s, es, n, en, m, em;
    two_prod(x.a, y.a, p, e);
    two_prod(x.a, y.b, q, eq);
    two_prod(x.b, y.a, s, es);
    two_sum(q, s, n, en);
    two_sum(n, e, m, em);
    float l = add(add(en, em), add(eq, es));
    l = fma(x.b, y.b, l);
    l = fma(x.a, y.c, l);
    l = fma(x.c, y.a, l);
    return W3{p, m, l};
}
VPMC_WIDE_FN W3 sqr3(const W3& x) {
    float p, e, m, em, n, en;
    const float x2 = add(x.a, x.a);
    two_prod(x.a, x.a, p, e);
    two_prod(x2, x.b, m, em);
    two_sum(m, e, n, en);
    float l = add(en, em);
    l = fma(x.b, x.b, l);
    l = fma(x2, x.c, l);
    return W3{p, n, l};
}
VPMC_WIDE_FN W3 norm3(const W3& x) {
    float a, b, t, c;
    fast_two_sum(x.a, x.b, a, t);
    fast_two_sum(t, x.c, b, c);
    return W3{a, b, c};
}
VPMC_WIDE_FN W3 sub3(const W3& x, const W3& y) {
    float s, e, m, em, n, en;
    two_sum(x.a, -y.a, s, e);
    two_sum(x.b, -y.b, m, em);
    two_sum(m, e, n, en);
    return W3{s, n, add(add(em, en), sub(x.c, y.c))};
}

// x + y (unnormalised).
VPMC_WIDE_FN W3 add3(const W3& x, const W3& y) {
    float s, e, m, em, n, en;
    two_sum(x.a, y.a, s, e);
    two_sum(x.b, y.b, m, em);
    two_sum(m, e, n, en);
    return W3{s, n, add(add(em, en), add(x.c, y.c))};
}
// (h + l) y and w y for single floats h, l, w.
VPMC_WIDE_FN W3 mul2(float h, float l, const W3& y) {
    float p, e, q, eq, s, es, n, en, m, em;
    two_prod(h, y.a, p, e);
    two_prod(h, y.b, q, eq);
    two_prod(l, y.a, s, es);
    two_sum(q, s, n, en);
    two_sum(n, e, m, em);
    float c = add(add(en, em), add(eq, es));
    c = fma(l, y.b, c);
    return W3{p, m, fma(h, y.c, c)};
}
VPMC_WIDE_FN W3 mul1(float w, const W3& y) {
    float p, e, q, eq, n, en;
    two_prod(w, y.a, p, e);
    two_prod(w, y.b, q, eq);
    two_sum(q, e, n, en);
    return W3{p, n, fma(w, y.c, add(en, eq))};
}
// 1 / x: the estimate y, then y (1 + e + e^2) with the residual e = 1 - x y to 2^-70.
VPMC_WIDE_FN W3 rcp3(const W3& x) {
    const float y = rcp_est(x.a);
    float f, fe, eh, el, p, pe;
    two_prod(x.b, y, f, fe);
    two_sum(fma(-x.a, y, 1.f), -f, eh, el);
    el = fma(-x.c, y, sub(el, fe));
    two_prod(y, eh, p, pe);
    return W3{y, p, fma(y, fma(eh, eh, el), pe)};
}

// |d|^2 of d = (xh + xl, yh + yl), |xl| <= ulp(xh); LOW = false: xl = yl = 0.
template <bool LOW>
VPMC_WIDE_FN W3 norm2(float xh, float xl, float yh, float yl) {
    float s, e, m, em, n, en;
    if (LOW) {
        const W3 x = sqr3(W3{xh, xl, 0.f}), y = sqr3(W3{yh, yl, 0.f});
        two_sum(x.a, y.a, s, e);
        two_sum(x.b, y.b, m, em);
        two_sum(m, e, n, en);
        return norm3(W3{s, n, add(add(em, en), add(x.c, y.c))});
    }
    float px, ex, py, ey;
    two_prod(xh, xh, px, ex);
    two_prod(yh, yh, py, ey);
    two_sum(px, py, s, e);
    two_sum(ex, ey, m, em);
    two_sum(m, e, n, en);
    return norm3(W3{s, n, add(em, en)});
}

// sqrt(x): the estimate g = x y (y ~ 1 / sqrt x), then g + rho / (2 g) - rho^2 / (8 g^3)
// with the residual rho = x - g^2 exact to 2^-70 and 1 / g = y (1 + eps), eps = 1 - y g.
VPMC_WIDE_FN W3 sqrt3(const W3& x) {
    const float y = rsqrt_est(x.a > 1e-30f ? x.a : 1e-30f);
    const float g = mul(x.a, y), hy = mul(0.5f, y);
    float gg, ge, a, e1, b, e2;
    two_prod(g, g, gg, ge);
    two_sum(sub(x.a, gg), -ge, a, e1);
    two_sum(a, x.b, b, e2);
    const float l = add(add(e1, e2), x.c);
    const float eps = fma(-y, g, 1.f);
    const float c0 = mul(b, hy);
    float c1 = fma(l, hy, fma(b, hy, -c0));
    c1 = fma(c0, eps, c1);
    c1 = fma(-mul(c0, c0), hy, c1);
    return norm3(W3{g, c0, c1});
}

// x added to a sum of three floats, which keeps more digits than an FP64 sum does.
VPMC_WIDE_FN void add_float(float (&s)[3], float x) {
    float e, f;
    two_sum(s[0], x, s[0], e);
    two_sum(s[1], e, s[1], f);
    s[2] = add(s[2], f);
}

// h^3 W(r) / (2 sigma) of the cubic spline at r^2 = r2 < h^2 (h a float, half_h3 =
// h^3 / 2 as a wide number): with t = h - r,
//   r > h / 2:   t^3
//   r <= h / 2:  h^3 / 2 - 3 r^2 t
// Below 0 (r a rounding above h) the result is to be dropped by its sign.
VPMC_WIDE_FN W3 spline_h3(const W3& r2, float h, const W3& half_h3) {
    const W3 r = sqrt3(r2);
    float t0, e, t1, f;
    fast_two_sum(h, -r.a, t0, e);
    two_sum(e, -r.b, t1, f);
    const W3 t = norm3(W3{t0, t1, sub(f, r.c)});
    if (add(t.a, t.a) >= h) {   // r <= h / 2
        const W3 p = norm3(mul3(r2, t));
        float a, b, c, d, n, en;
        two_prod(3.f, p.a, a, b);
        two_prod(3.f, p.b, c, d);
        two_sum(c, b, n, en);
        return sub3(half_h3, W3{a, n, fma(3.f, p.c, add(d, en))});
    }
    return mul3(sqr3(t), t);
}

// acc += w v, w = w0 + w1.
VPMC_WIDE_FN void add_product(W3& acc, float w0, float w1, const W3& v) {
    float z, ez, p, ep, q, eq, m, em, n, en, s, es, k, ek, o, eo;
    two_prod(w0, v.a, z, ez);
    two_prod(w0, v.b, p, ep);
    two_prod(w1, v.a, q, eq);
    two_sum(p, q, m, em);
    two_sum(m, ez, n, en);
    float l = add(add(em, en), add(ep, eq));
    l = fma(w0, v.c, l);
    l = fma(w1, v.b, l);
    two_sum(acc.a, z, s, es);
    two_sum(acc.b, n, k, ek);
    two_sum(k, es, o, eo);
    acc.c = add(l, add(add(ek, eo), acc.c));
    fast_two_sum(s, o, acc.a, acc.b);
}

}  // namespace wide
}  // namespace vpmc
