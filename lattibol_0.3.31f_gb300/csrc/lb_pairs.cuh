// lb_pairs.cuh -- the native arithmetic on two nodes at once, one in each lane
// of the paired FP32 instructions (.f32x2).  Every lane performs the scalar
// form's operations in the scalar form's order, so the bits are the same.  The
// paired instructions issue at half the rate of the scalar ones (0.47 against
// 0.90 per clock and scheduler, measured): they halve the issue slots, not the
// FP32 pipe's time.
#pragma once

#include "lb_kernels.cuh"

namespace lb {

__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }

// The constants of the paired forms, each twice: the instructions read them as
// register pairs or 8-byte constant operands.  one and mone (+1, -1) stand in
// sums of products: a product that feeds a paired addition is contracted with
// it by the assembler, a fused multiply-add by a factor the compiler does not
// know is not.
struct PairConst {
    float2 one, mone, c45, c3, m3, m15;
};
inline PairConst pair_constants() {
    const auto two = [](float v) { return make_float2(v, v); };
    return PairConst{two(1.f), two(-1.f), two(4.5f), two(3.f), two(-3.f), two(-1.5f)};
}
__device__ __forceinline__ float2 pair_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 pair_sub(const PairConst &c, float2 a, float2 b) {
    return __ffma2_rn(b, c.mone, a);
}
// a + b where an operand is a product
__device__ __forceinline__ float2 pair_addp(const PairConst &c, float2 a, float2 b) {
    return __ffma2_rn(b, c.one, a);
}

// 1 / x of both lanes, correctly rounded: the hardware approximation (within 1
// ulp) and one Newton step whose residual e = 1 - x y and update y + y e are
// single fused roundings, which Markstein's theorem (Markstein, "Computation
// of elementary functions on the IBM RISC System/6000 processor", 1990) makes
// the correctly rounded reciprocal.  The same bits as 1.f / x on all 2^32
// arguments (tests/test_gpu_every_float.py); where the residual says that the
// approximation is none (zero, infinite, NaN or subnormal x or 1 / x) the
// divisions themselves run.  9 issue slots for the two lanes, against about 45
// for two divisions and the moves around them.
__device__ __forceinline__ float2 pair_rcp(const PairConst &c, float2 x) {
    float2 y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y.x) : "f"(x.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y.y) : "f"(x.y));
    const float2 m = __fmul2_rn(x, c.mone);
    const float2 e = __ffma2_rn(m, y, c.one);
    if (fabsf(e.x) + fabsf(e.y) < 0.5f) return __ffma2_rn(y, e, y);
    return make_float2(1.f / x.x, 1.f / x.y);
}

// two reciprocals at once (a check for both)
__device__ __forceinline__ void pair_rcp2(const PairConst &c, float2 &x, float2 &y) {
    float2 p, q;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(p.x) : "f"(x.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(p.y) : "f"(x.y));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(q.x) : "f"(y.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(q.y) : "f"(y.y));
    const float2 e = __ffma2_rn(__fmul2_rn(x, c.mone), p, c.one);
    const float2 f = __ffma2_rn(__fmul2_rn(y, c.mone), q, c.one);
    if ((fabsf(e.x) + fabsf(e.y)) + (fabsf(f.x) + fabsf(f.y)) < 0.5f) {
        x = __ffma2_rn(p, e, p);
        y = __ffma2_rn(q, f, q);
        return;
    }
    x = make_float2(1.f / x.x, 1.f / x.y);
    y = make_float2(1.f / y.x, 1.f / y.y);
}

// the step's physics in paired form: -w0, -w1, -w5, -tau_inv, tau_inv, force
struct PairD2 {
    float2 n0, n1, n5, mt, tau, Fx, Fy;
};

// psi = 1 - exp(-rho) of both lanes: psi_exp1's operations (lb_expf for |x| <= 87,
// the scalar form beyond; the first product of its reduction is exact, so its
// subtraction may be fused)
__device__ __forceinline__ float2 pair_psi_exp1(const PairConst &c, float2 rho) {
    const float2 x = __fmul2_rn(rho, c.mone);
    const float2 s = __ffma2_rn(__fmul2_rn(x, both(0x1.715476p+0f)), c.one, both(0x1.8p+23f));
    const float2 k = pair_add(s, both(-0x1.8p+23f));
    const float2 d = __ffma2_rn(k, both(-0x1.62ep-1f), x);
    const float2 r = __ffma2_rn(__fmul2_rn(k, both(0x1.0bfbe8p-15f)), c.mone, d);
    float2 p = both(0x1.a01a02p-13f);
    const auto horner = [&](float a) { p = __ffma2_rn(__fmul2_rn(p, r), c.one, both(a)); };
    horner(0x1.6c16c2p-10f);
    horner(0x1.111112p-7f);
    horner(0x1.555556p-5f);
    horner(0x1.555556p-3f);
    horner(0.5f);
    horner(1.0f);
    horner(1.0f);
    const float2 two_k = make_float2(__int_as_float((__float_as_int(s.x) << 23) + 0x3f800000),
                                     __int_as_float((__float_as_int(s.y) << 23) + 0x3f800000));
    const float2 psi = __ffma2_rn(__fmul2_rn(p, two_k), c.mone, c.one);
    if (fabsf(x.x) <= 87.f && fabsf(x.y) <= 87.f) return psi;
    return make_float2(psi_exp1(rho.x), psi_exp1(rho.y));
}

// d2q9_moments_native of two nodes
__device__ __forceinline__ void d2q9_moments_pairs(const PairConst &c, const float2 (&g)[9],
                                                   float2 &rho, float2 &ux, float2 &uy) {
    const auto add = [](float2 a, float2 b) { return pair_add(a, b); };
    const float2 px = add(add(g[1], g[5]), g[8]);
    const float2 mx = add(add(g[3], g[6]), g[7]);
    const float2 zx = add(add(g[0], g[2]), g[4]);
    rho = add(add(px, mx), zx);
    const float2 jy = pair_sub(c, add(add(g[2], g[5]), g[6]), add(add(g[4], g[7]), g[8]));
    const float2 inv = pair_rcp(c, rho);
    ux = __fmul2_rn(pair_sub(c, px, mx), inv);
    uy = __fmul2_rn(jy, inv);
}

// d2q9_bgk_native of two nodes
__device__ __forceinline__ void d2q9_bgk_pairs(const PairConst &c, const PairD2 &d,
                                               float2 (&g)[9], float2 ex, float2 ey, float2 rho) {
    const float2 usq = __ffma2_rn(ey, ey, __fmul2_rn(ex, ex));
    const float2 base = __ffma2_rn(c.m15, usq, c.one);
    // e = -(f_eq - g) in one rounding, then g - tau_inv e: the scalar form with
    // both signs turned (rounding is symmetric)
    const float2 n0 = __fmul2_rn(d.n0, rho), n1 = __fmul2_rn(d.n1, rho),
                 n5 = __fmul2_rn(d.n5, rho);
    g[0] = __ffma2_rn(d.mt, __ffma2_rn(n0, base, g[0]), g[0]);
    auto pair = [&](int kp, int km, float2 n, float2 p) {
        const float2 t = __ffma2_rn(__fmul2_rn(c.c45, p), p, base);
        g[kp] = __ffma2_rn(d.mt, __ffma2_rn(n, __ffma2_rn(c.c3, p, t), g[kp]), g[kp]);
        g[km] = __ffma2_rn(d.mt, __ffma2_rn(n, __ffma2_rn(c.m3, p, t), g[km]), g[km]);
    };
    pair(1, 3, n1, ex);
    pair(2, 4, n1, ey);
    pair(5, 7, n5, pair_addp(c, ex, ey));
    pair(6, 8, n5, pair_sub(c, ey, ex));
}

// d2q9_collide_native of two nodes (force: Fx or Fy is not zero)
__device__ __forceinline__ void d2q9_collide_pairs(const PairConst &c, const PairD2 &d,
                                                   float2 (&g)[9], bool force, float2 &rho,
                                                   float2 &ux, float2 &uy) {
    d2q9_moments_pairs(c, g, rho, ux, uy);
    float2 ex = ux, ey = uy;
    if (force) {
        const float2 irt = pair_rcp(c, __fmul2_rn(rho, d.tau));
        if (d.Fx.x != 0.f) ex = __ffma2_rn(d.Fx, irt, ux);
        if (d.Fy.x != 0.f) ey = __ffma2_rn(d.Fy, irt, uy);
    }
    d2q9_bgk_pairs(c, d, g, ex, ey, rho);
}

// a row's column pairs (lane l: columns 2l, 2l + 1) read one column to the left
// (c = +1: the value that moves in from x - 1) or to the right (c = -1)
__device__ __forceinline__ float2 row_shift(float2 v, int c) {
    if (c > 0) return make_float2(__shfl_up_sync(0xffffffffu, v.y, 1), v.x);
    if (c < 0) return make_float2(v.y, __shfl_down_sync(0xffffffffu, v.x, 1));
    return v;
}

}  // namespace lb
