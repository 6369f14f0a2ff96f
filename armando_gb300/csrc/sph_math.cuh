// sph_math.cuh -- per-pair arithmetic of the fused SPH passes.
//
// Compiles as CUDA device code and as plain C++ (host shims below), so the
// exact FP32 operation sequence of the kernels can be replayed on a CPU.
//
// Formulas:
//   Wendland C2 (ArmandoThrust/armando.cu:137-191; 2D constant acpu.c:162):
//     W      = K_dim / h^dim * (1 - q/2)^4 (1 + 2q),          q = r / h
//     dW/dx  = K_dim * 5/8 / h^(dim+2) * (q - 2)^3 * (x_i - x_j)
//     K_2 = 7/(4 pi), K_3 = 21/(16 pi) (15/(16 pi) with the legacy switch)
//   Pair test (CERNsource/link_list.f:154-159): dr^2 < (h_i + h_j)^2 with dr^2
//     summed over axes in order, no fused multiply-add, so neighbour sets are
//     bit-identical to the FP32 link_list of the oracle.
//   Tait (FORTRANsource/eos.f90:255-283): p = rho0 c0^2/7 ((1+d)^7 - 1),
//     d = (rho - rho0)/rho0, evaluated as the exact binomial polynomial in d.
#pragma once

#if defined(__CUDACC__)
#define SPH_HD __device__ __forceinline__
#else
#include <cmath>
#define SPH_HD inline
// Host stand-ins for the round-to-nearest intrinsics (build with -ffp-contract=off).
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fdiv_rn(float a, float b) { return a / b; }
inline float __frcp_rn(float a) { return 1.0f / a; }
inline float __fsqrt_rn(float a) { return std::sqrt(a); }
inline float rsqrtf(float a) { return 1.0f / std::sqrt(a); }
#endif

namespace sph {

// ---- float-float (unevaluated sum hi + lo) helpers: error-free transforms ----
struct ff {
    float hi, lo;
};

// Knuth TwoSum: s + e == a + b exactly.
SPH_HD ff two_sum(float a, float b) {
    float s = __fadd_rn(a, b);
    float bb = __fsub_rn(s, a);
    float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    return {s, e};
}
// a - b == s + e exactly (TwoSum of a and -b).
SPH_HD ff two_diff(float a, float b) {
    float s = __fsub_rn(a, b);
    float bb = __fsub_rn(s, a);
    float e = __fsub_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fadd_rn(b, bb));
    return {s, e};
}
// a * b == p + e exactly (fused multiply-add residual).
SPH_HD ff two_prod(float a, float b) {
    float p = __fmul_rn(a, b);
    float e = fmaf(a, b, -p);
    return {p, e};
}
// (a.hi + a.lo) * (b.hi + b.lo), relative error ~2^-44.
SPH_HD ff ff_mul(ff a, ff b) {
    ff p = two_prod(a.hi, b.hi);
    p.lo = fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, p.lo));
    return p;
}
SPH_HD ff ff_mul_f(ff a, float b) {
    ff p = two_prod(a.hi, b);
    p.lo = fmaf(a.lo, b, p.lo);
    return p;
}
SPH_HD ff ff_sqr(ff a) {
    ff p = two_prod(a.hi, a.hi);
    p.lo = fmaf(__fmul_rn(2.0f, a.hi), a.lo, p.lo);
    return p;
}
// Accumulate x into acc (acc.lo collects every rounding error).
SPH_HD void ff_acc(ff& acc, ff x) {
    ff s = two_sum(acc.hi, x.hi);
    acc.hi = s.hi;
    acc.lo = __fadd_rn(acc.lo, __fadd_rn(s.lo, x.lo));
}

// 1/h as float-float: Newton residual of the correctly rounded reciprocal.
SPH_HD ff ff_recip(float h) {
    float r = __frcp_rn(h);
    float e = fmaf(-r, h, 1.0f);  // exact: 1 - r*h
    return {r, __fmul_rn(e, r)};
}

// ---- Pair test (bit-exact mirror of the oracle's FP32 link_list) ----
template <int DIM>
SPH_HD float dist2_exact(const float* d) {
    float s = __fmul_rn(d[0], d[0]);
    s = __fadd_rn(s, __fmul_rn(d[1], d[1]));
    if (DIM == 3) s = __fadd_rn(s, __fmul_rn(d[2], d[2]));
    return s;
}
SPH_HD bool within_support(float dr2, float hi, float hj) {
    float s = __fadd_rn(hi, hj);
    return dr2 < __fmul_rn(s, s);
}
// Minimum image on a periodic axis, same branch order as the oracle.
SPH_HD float min_image(float dx, float L, float half) {
    if (dx > half) return __fsub_rn(dx, L);
    if (dx < -half) return __fadd_rn(dx, L);
    return dx;
}

// Tait pressure from d = rho/rho0 - 1: B * ((1+d)^7 - 1), B = rho0 c0^2 / 7.
SPH_HD float tait_poly(float d, float B) {
    float y = __fadd_rn(7.0f, d);
    y = fmaf(y, d, 21.0f);
    y = fmaf(y, d, 35.0f);
    y = fmaf(y, d, 35.0f);
    y = fmaf(y, d, 21.0f);
    y = fmaf(y, d, 7.0f);
    return __fmul_rn(B, __fmul_rn(y, d));
}

}  // namespace sph
