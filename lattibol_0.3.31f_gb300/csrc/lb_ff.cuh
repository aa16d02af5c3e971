// lb_ff.cuh -- the reference's FP64 lines in pairs of floats.
//
// The reference mode promotes two places to FP64 (its double literals): the
// pseudo-potential 4 exp(-200 / rho) and the Zou-He faces.  This GPU runs two
// FP64 operations per clock and SM, a sixty-fourth of its FP32 rate: psi of a
// 704 x 440 lattice took 18.5 us (4.2 us to copy the same values), the whole
// collision pass 24 us with the FP64 pipe 74 % busy.  Every one of these lines
// ends in a rounding to float, so the value is formed here as an unevaluated
// sum of two floats with a known error bound, and rounded.  Where both ends of
// the bound round to the same float that is the float the FP64 line gives (its
// own error is far below the bound); elsewhere, and outside the range the
// bound was made for, the FP64 line itself runs.  Same bits, on every input.
#pragma once

#include <cmath>

#include <cuda_runtime.h>

namespace lb {

// a + b = s + e exactly (Knuth)
__device__ __forceinline__ float ff_sum(float a, float b, float &e) {
    const float s = a + b, t = s - a;
    e = (a - (s - t)) + (b - t);
    return s;
}
// a b = p + e exactly
__device__ __forceinline__ float ff_mul(float a, float b, float &e) {
    const float p = a * b;
    e = __fmaf_rn(a, b, -p);
    return p;
}
// the float nearest to s + lo, known to within `bound`: false when the bound
// does not decide it (or the value is so small that its parts may be subnormal)
__device__ __forceinline__ bool ff_round(float s, float lo, float bound, float &out) {
    out = s + (lo + bound);
    return out == s + (lo - bound) && fabsf(out) > 1e-28f;
}

// 1 / x within 1 ulp, from the hardware (a host model of these forms brings its own)
#ifdef __CUDACC__
__device__ __forceinline__ float ff_rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
#else
float ff_rcp(float x);
#endif

// a positive constant as two floats (48 bits)
struct FF {
    float hi, lo;
};
__host__ __device__ constexpr FF ff_const(double v) {
    return FF{(float)v, (float)(v - (double)(float)v)};
}
// 1 / v as two floats, for ff_ratio.  The low part of a quotient below 2^-100 may
// lie among the subnormal floats and keep fewer bits than ff_ratio's bound allows
// for (v = 1e34: 1 result in 26 rounded the wrong way); such a pair is not a
// number, on which ff_ratio leaves the value to the FP64 line.
inline FF ff_reciprocal(double v) {
    const double r = 1. / v;
    if (r < 0x1p-100 && r > -0x1p-100) return FF{NAN, NAN};
    return ff_const(r);
}

// 4 exp(-200 / rho) rounded to float, for rho in [8, 2^20].  The quotient by its
// exact remainder (relative error 2^-46); reduction by k ln 2 with ln 2 in three
// parts (Cody and Waite's scheme; the first part has 16 bits, so k times it is
// exact); the Taylor polynomial of degree 10, its last five steps in pairs of
// floats.  Relative error: the series' remainder r^11 / 11! is at most 2^-42 for
// |r| <= 0.35, the single-float sum p of the terms from r^5 / 5! on carries about
// 2^-37 of the result, everything else below 2^-39.  Found on all 142 606 337
// floats of the range, with the reciprocal's seed off by -1, 0 and +1 ulp: at most
// 2^-36.8 against 64-bit arithmetic (with degree 9, whose remainder is 2^-36.6:
// 2^-35.7).  The bound is 2^-35, 3.5 times that; about one value in 1200 takes the
// FP64 line.
// the value as hi + lo; false outside the range
__device__ __forceinline__ bool ff_psi_parts(float rho, float &hi, float &lo) {
    if (!(rho >= 8.f && rho <= 1048576.f)) return false;
    float y = ff_rcp(rho);
    y = __fmaf_rn(y, __fmaf_rn(-rho, y, 1.f), y);
    const float q = -200.f * y;
    const float q_lo = __fmaf_rn(-q, rho, -200.f) * y;  // exact remainder over rho
    const float s = q * 0x1.715476p+0f + 0x1.8p+23f;     // k in the low bits
    const float k = s - 0x1.8p+23f;
    // ln 2 = 0x1.62e4p-1 + 0x1.7f7d1cp-20 + 0x1.ef35794p-45
    const float rh0 = __fmaf_rn(-k, 0x1.62e4p-1f, q);    // exact
    float m_lo, e1, e2;
    const float m = ff_mul(k, 0x1.7f7d1cp-20f, m_lo);
    const float t = ff_sum(q_lo, -m, e1);
    const float rh = ff_sum(rh0, t, e2);
    const float rl = e2 + (e1 - __fmaf_rn(k, 0x1.ef3578p-45f, m_lo));
    // 1/4! + r (1/5! + ... + r^5 / 10!), the sum with 1/4! in two floats
    float p = 0x1.27e4fcp-22f;
    p = __fmaf_rn(p, rh, 0x1.71de3ap-19f);
    p = __fmaf_rn(p, rh, 0x1.a01a02p-16f);
    p = __fmaf_rn(p, rh, 0x1.a01a02p-13f);
    p = __fmaf_rn(p, rh, 0x1.6c16c2p-10f);
    p = __fmaf_rn(p, rh, 0x1.111112p-7f);
    float h = 0x1.555556p-5f, l = -0x1.555556p-30f;      // 1/24
    {
        const float u = __fmaf_rn(p, rh, h);
        l = (__fmaf_rn(p, rh, h - u)) + l;
        h = u;
    }
    // h + l := c + (rh + rl)(h + l)
    auto step = [&](float c, float c_lo) {
        float e;
        const float u = ff_mul(rh, h, e);
        e = __fmaf_rn(rl, h, __fmaf_rn(rh, l, e));
        const float v = c + u;
        l = ((c - v) + u) + (e + c_lo);
        h = v;
    };
    step(0x1.555556p-3f, -0x1.555556p-28f);  // 1/6
    step(0.5f, 0.f);
    step(1.f, 0.f);
    step(1.f, 0.f);
    const float scale = __int_as_float((__float_as_int(s) << 23) + 0x40800000);  // 4 * 2^k
    hi = h * scale;
    lo = l * scale;
    return true;
}
__device__ __forceinline__ bool ff_psi_ref(float rho, float &out) {
    float h, l;
    return ff_psi_parts(rho, h, l) && ff_round(h, l, 0x1p-35f * h, out);
}

// (float)((double)base + c (double)ru - 0.5 (double)t2): one line of the Zou-He
// faces (t2 = 0: the two-term lines)
__device__ __forceinline__ bool ff_face(float base, FF c, float ru, float t2, float &out) {
    float e0, e1, e2;
    const float p = ff_mul(c.hi, ru, e0);
    e0 = __fmaf_rn(c.lo, ru, e0);
    const float h = 0.5f * t2;
    const float s1 = ff_sum(base, p, e1);
    const float s2 = ff_sum(s1, -h, e2);
    return ff_round(s2, (e1 + e2) + e0, 0x1p-42f * (fabsf(base) + fabsf(p) + fabsf(h)), out);
}

// (float)(add + ((double)a + 2 (double)b) inv), inv = 1 / (1 - ux) or 1 / rho_out
// to 48 bits (ff_reciprocal): the density and velocity of a Zou-He face
__device__ __forceinline__ bool ff_ratio(float a, float b, FF inv, float add, float &out) {
    float e0, e1, e2;
    const float n = ff_sum(a, 2.f * b, e0);
    const float p = ff_mul(n, inv.hi, e1);
    e1 = __fmaf_rn(n, inv.lo, __fmaf_rn(e0, inv.hi, e1));
    const float s = ff_sum(add, p, e2);
    return ff_round(s, e2 + e1, 0x1p-44f * (fabsf(add) + fabsf(p)), out);
}

}  // namespace lb
