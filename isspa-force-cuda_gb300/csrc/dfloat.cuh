// dfloat.cuh -- double-float arithmetic: a value carried as the unevaluated sum
// of two FP32 words, about 48 significant bits on the FP32 pipe.
#pragma once
#include <cuda_runtime.h>

namespace isspa {
namespace {

// Double-float values (hi + lo, two FP32 words) from the error-free
// transformations of Knuth (TwoSum) and Dekker (TwoProduct, here with an FMA):
// the bond stretch r0 - |r| and the angle bend theta - theta0 of a geometry
// near its minimum are small differences of O(1) quantities, which FP32 alone
// resolves only to ~1e-7 absolute (a relative error of the force that grows
// as the force vanishes).  Carried in double-float they keep ~1e-7 of their
// own size; every operation is an FP32 instruction (__fadd_rn / __fmul_rn /
// fmaf, never contracted or reassociated).
struct DF {
    float hi, lo;
};
__device__ __forceinline__ DF two_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    return DF{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
__device__ __forceinline__ DF fast_two_sum(float a, float b) {  // |a| >= |b|
    const float s = __fadd_rn(a, b);
    return DF{s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ DF two_prod(float a, float b) {
    const float p = __fmul_rn(a, b);
    return DF{p, fmaf(a, b, -p)};
}
__device__ __forceinline__ DF df_add(DF a, DF b) {
    const DF s = two_sum(a.hi, b.hi);
    return fast_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}
__device__ __forceinline__ DF df_neg(DF a) { return DF{-a.hi, -a.lo}; }
__device__ __forceinline__ DF df_mul(DF a, DF b) {
    const DF p = two_prod(a.hi, b.hi);
    return fast_two_sum(p.hi, fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, p.lo)));
}
__device__ __forceinline__ DF df_sqrt(DF a) {  // a > 0; one Newton step on the FP32 root
    const float s = __fsqrt_rn(a.hi);
    const float res = __fadd_rn(fmaf(-s, s, a.hi), a.lo);
    return fast_two_sum(s, __fdiv_rn(res, __fmul_rn(2.0f, s)));
}
__device__ __forceinline__ float df_float(DF a) { return __fadd_rn(a.hi, a.lo); }

// DF times a float, and the exact product of a small integer scale
__device__ __forceinline__ DF df_mulf(DF a, float b) {
    const DF p = two_prod(a.hi, b);
    return fast_two_sum(p.hi, fmaf(a.lo, b, p.lo));
}
__device__ __forceinline__ DF df_addf(DF a, float b) {
    const DF s = two_sum(a.hi, b);
    return fast_two_sum(s.hi, __fadd_rn(s.lo, a.lo));
}
// a times a power of two
__device__ __forceinline__ DF df_scale(DF a, float p) { return DF{__fmul_rn(a.hi, p), __fmul_rn(a.lo, p)}; }
// a b + c
__device__ __forceinline__ DF df_fma(DF a, DF b, DF c) { return df_add(df_mul(a, b), c); }
// x^2 + y^2 + z^2 (the compensated dot product of Ogita, Rump & Oishi 2005)
__device__ __forceinline__ DF df_norm2(float x, float y, float z) {
    const DF a = two_prod(x, x), b = two_prod(y, y), c = two_prod(z, z);
    const DF s = two_sum(a.hi, b.hi), t = two_sum(s.hi, c.hi);
    return fast_two_sum(t.hi, (s.lo + t.lo) + ((a.lo + b.lo) + c.lo));
}
// 1/sqrt(a), a > 0: one Newton step on the FP32 reciprocal root, its residual in
// double-float
__device__ __forceinline__ DF df_rsqrt(DF a) {
    const float y = rsqrtf(a.hi);
    const DF q = df_mul(a, two_prod(y, y));
    const float e = __fsub_rn(__fsub_rn(1.0f, q.hi), q.lo);  // 1 - a y^2 (q.hi is near 1)
    return fast_two_sum(y, __fmul_rn(__fmul_rn(0.5f, y), e));
}
// sqrt(a) from the FP32 reciprocal root; 0 for a = 0
__device__ __forceinline__ DF df_root(DF a) {
    const float y = a.hi > 0.0f ? rsqrtf(a.hi) : 0.0f;
    const float s = __fmul_rn(a.hi, y);
    return fast_two_sum(s, __fmul_rn(__fadd_rn(fmaf(-s, s, a.hi), a.lo), __fmul_rn(0.5f, y)));
}
// a / b: an FP32 quotient and the quotient of its residual
__device__ __forceinline__ DF df_div(DF a, DF b) {
    const float inv = __fdividef(1.0f, b.hi);
    const float q = __fmul_rn(a.hi, inv);
    const DF p = two_prod(b.hi, q);
    const float r = __fadd_rn(__fsub_rn(__fsub_rn(a.hi, p.hi), p.lo), fmaf(-b.lo, q, a.lo));
    return fast_two_sum(q, __fmul_rn(r, inv));
}
// ((a - r0) inv) - bin for a table bin that holds a: the last difference is exact
__device__ __forceinline__ DF df_table_frac(DF a, float r0, DF inv, int bin) {
    const DF t = two_sum(a.hi, -r0);
    const DF p = two_prod(t.hi, inv.hi);
    const float lo = fmaf(t.hi, inv.lo, fmaf(__fadd_rn(t.lo, a.lo), inv.hi, p.lo));
    return fast_two_sum(__fsub_rn(p.hi, (float)bin), lo);
}
// v0 + f (v1 - v0)
__device__ __forceinline__ DF df_lerp(float v0, float v1, DF f) {
    const DF d = two_sum(v1, -v0);
    const DF p = two_prod(d.hi, f.hi);
    const DF s = two_sum(v0, p.hi);
    return fast_two_sum(s.hi, __fadd_rn(s.lo, fmaf(d.hi, f.lo, fmaf(d.lo, f.hi, p.lo))));
}
__device__ __forceinline__ DF df_from(double v) {
    const float hi = (float)v;
    return DF{hi, (float)(v - (double)hi)};
}
__device__ __forceinline__ double df_double(DF a) { return (double)a.hi + (double)a.lo; }

}  // namespace
}  // namespace isspa
