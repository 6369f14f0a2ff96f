// pair2.cuh -- two neighbours of a particle at a time in packed FP32.
//
// sm_103 executes an FP32 instruction on a register pair (two values) in two
// cycles of the FMA pipe but one issue slot. The neighbour passes were bound by
// issue (a list entry's address, loads, comparisons and reciprocals share the
// slots with its arithmetic), so their pair arithmetic runs on two entries at
// once. Every operation below is an explicit rounding: all instantiations of a
// pass round alike, whatever the compiler contracts elsewhere.
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
__device__ __forceinline__ f2 rsqrt2(f2 a) { return make_float2(rsqrt_fast(a.x), rsqrt_fast(a.y)); }

// Added to squared distances before a reciprocal square root: no effect on any
// distance above 1e-15 times the unit, and a coincident pair (or a particle
// with itself) gets r = 0 without a comparison.
constexpr float kTinyDr2 = 1.0e-37f;

}  // namespace ag
