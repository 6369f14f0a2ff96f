// pair2.cuh -- two neighbours of a particle at a time in packed FP32.
//
// sm_103 executes an FP32 instruction on a register pair (two values) in two
// cycles of the FMA pipe but one issue slot. The neighbour passes were bound by
// issue (a list entry's address, loads, comparisons and reciprocals share the
// slots with its arithmetic), so their pair arithmetic runs on two entries at
// once. A packed product is fused with an addition that takes it (measured: also the
// .rn forms), unlike the scalar __fmul_rn; prod2 keeps its own rounding.
#pragma once

namespace ag {

using f2 = float2;

__device__ __forceinline__ f2 bc2(float a) { return make_float2(a, a); }
__device__ __forceinline__ f2 neg2(f2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ f2 mul2(f2 a, f2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ f2 add2(f2 a, f2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ f2 sub2(f2 a, f2 b) { return __fadd2_rn(a, neg2(b)); }
__device__ __forceinline__ f2 max2(f2 a, float b) { return make_float2(fmaxf(a.x, b), fmaxf(a.y, b)); }
__device__ __forceinline__ f2 min2(f2 a, float b) { return make_float2(fminf(a.x, b), fminf(a.y, b)); }
// Added to squared distances before a reciprocal square root: no effect on any
// distance above 1e-15 times the unit, and a coincident pair (or a particle
// with itself) gets r = 0 without a comparison.
constexpr float kTinyDr2 = 1.0e-37f;
// a b rounded, also where an addition takes it (for results above 1e-29).
__device__ __forceinline__ f2 prod2(f2 a, f2 b) { return __ffma2_rn(a, b, make_float2(kTinyDr2, kTinyDr2)); }
// The x coordinate given to an absent entry (the odd end of a list, a lane whose list is
// shorter than its neighbours'), which otherwise repeats the particle itself: beyond
// every support, where the kernel's gradient is zero. At d = 0, where it is largest, the
// rounding of two products that should cancel, an infinite P or the quotient of a
// vanishing r^2 would stay.
constexpr float kOutOfReach = 1.0e18f;
// v where t < 0, else 0 (also in place of an infinity or NaN).
__device__ __forceinline__ f2 within2(f2 t, f2 v) {
    return make_float2(t.x < 0.f ? v.x : 0.f, t.y < 0.f ? v.y : 0.f);
}
// acc + a.x b.x + a.y b.y, in that order (one rounding per term).
__device__ __forceinline__ float dot2(f2 a, f2 b, float acc) { return fmaf(a.y, b.y, fmaf(a.x, b.x, acc)); }

// One-instruction reciprocal (square root): no handling of denormal inputs, which
// the callers keep out.
__device__ __forceinline__ float rcp_fast(float a) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ float rsqrt_fast(float a) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ f2 rcp2(f2 a) { return make_float2(rcp_fast(a.x), rcp_fast(a.y)); }
// 1 / (a b) for a b >= 0, finite also where the product vanishes (prod2's constant: no
// register pair of its own).
__device__ __forceinline__ f2 rcp_prod2(f2 a, f2 b) { return rcp2(prod2(a, b)); }
__device__ __forceinline__ f2 rsqrt2(f2 a) { return make_float2(rsqrt_fast(a.x), rsqrt_fast(a.y)); }

// ---- float-float on two values at once (hi + lo each; sph_math.cuh's forms) ----
struct ff2 {
    f2 hi, lo;
};
// Knuth TwoSum: hi + lo == a + b exactly.
__device__ __forceinline__ ff2 two_sum2(f2 a, f2 b) {
    const f2 s = add2(a, b), bb = sub2(s, a);
    return {s, add2(sub2(a, sub2(s, bb)), sub2(b, bb))};
}
__device__ __forceinline__ ff2 two_prod2(f2 a, f2 b) {
    const f2 p = mul2(a, b);
    return {p, fma2(a, b, neg2(p))};
}
__device__ __forceinline__ ff2 mul_ff2(ff2 a, ff2 b) {
    ff2 p = two_prod2(a.hi, b.hi);
    p.lo = fma2(a.hi, b.lo, fma2(a.lo, b.hi, p.lo));
    return p;
}
__device__ __forceinline__ ff2 mul_ff2_f(ff2 a, f2 b) {
    ff2 p = two_prod2(a.hi, b);
    p.lo = fma2(a.lo, b, p.lo);
    return p;
}
__device__ __forceinline__ ff2 sqr_ff2(ff2 a) {
    ff2 p = two_prod2(a.hi, a.hi);
    p.lo = fma2(add2(a.hi, a.hi), a.lo, p.lo);
    return p;
}
// c + k a for |c| >= |k a.hi| and k a power of two (Fast2Sum).
__device__ __forceinline__ ff2 fast_affine2(ff2 a, float k, float c) {
    const f2 s = fma2(a.hi, bc2(k), bc2(c));
    const f2 z = sub2(s, bc2(c));
    return {s, fma2(a.lo, bc2(k), fma2(a.hi, bc2(k), neg2(z)))};
}
// acc += x, every rounding error collected in the low part.
__device__ __forceinline__ void acc_ff2(f2& hi, f2& lo, ff2 x) {
    const ff2 s = two_sum2(hi, x.hi);
    hi = s.hi;
    lo = add2(lo, add2(s.lo, x.lo));
}
__device__ __forceinline__ void acc_ff2(f2& hi, f2& lo, f2 x) {
    const ff2 s = two_sum2(hi, x);
    hi = s.hi;
    lo = add2(lo, s.lo);
}

// ---- correctly rounded results (Markstein, "Computation of elementary functions on the
// IBM RISC System/6000 processor", 1990): an estimate and the exact FMA residual of the
// result, so the rounding differs from IEEE's at most where the exact value is within
// 2^-19 ulp of a tie: the estimates are off by 2^-22.4 at most, which the correction
// squares (4 million random operands of each: no difference). For operands and results
// far from the overflow and underflow limits (the estimates flush there).
// a / b; y: an estimate of 1/b.
__device__ __forceinline__ f2 div2(f2 a, f2 b, f2 y) {
    const f2 q = mul2(a, y);
    return fma2(fma2(neg2(b), q, a), y, q);
}
__device__ __forceinline__ f2 div2(f2 a, f2 b) { return div2(a, b, rcp2(b)); }
// 1 / b.
__device__ __forceinline__ f2 rcp2_rn(f2 b, f2 y) { return fma2(fma2(neg2(b), y, bc2(1.0f)), y, y); }
// 1/a as float-float: the rounded reciprocal and its exact residual (relative error below
// 2^-47; from the unrounded one 2^-46.2).
__device__ __forceinline__ ff2 recip_ff2(f2 a) {
    const f2 r = rcp2_rn(a, rcp2(a));
    return {r, mul2(r, fma2(neg2(r), a, bc2(1.0f)))};
}
// sqrt(a); y: an estimate of 1/sqrt(a).
__device__ __forceinline__ f2 sqrt2(f2 a, f2 y) {
    const f2 r = mul2(a, y);
    return fma2(fma2(neg2(r), r, a), mul2(y, bc2(0.5f)), r);
}

// sqrt: the hardware reciprocal square root and one Newton correction from the exact
// residual a.hi - r^2 (relative error ~2^-44). 0 for a = 0.
__device__ __forceinline__ ff2 sqrt_ff2(ff2 a) {
    const f2 rs = rsqrt2(max2(a.hi, kTinyDr2));
    const f2 r = mul2(a.hi, rs);
    const f2 res = add2(fma2(neg2(r), r, a.hi), a.lo);
    return {r, mul2(res, mul2(rs, bc2(0.5f)))};
}

}  // namespace ag
