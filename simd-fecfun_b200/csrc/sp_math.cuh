// tanh(a/2) and 2 atanh(m) of the sum-product update, written without
// branches: the same values, bit for bit, as the functions of ldpc_math.h,
// for the arguments that the update produces (a >= 0; 0 <= m <= 1, NaN for
// m = 1 as there).
//
// Why a second form.  The update evaluates both functions on every edge.  In
// ldpc_math.h each has two series behind a branch that a warp's lanes split
// on, and correctly rounded divisions, each with a call for out-of-range
// operands; the compiler can neither interleave the chains of several edges
// across those branches nor skip either side (802.16e Z = 96: 307 warp
// instructions per edge, "wait" the first stall).  Here
//   - both series are one Horner chain on a selected argument: e^y - 1 for
//     small |y| has the coefficients of e^r, one step further along;
//   - a division is a reciprocal approximation, Newton's step, the quotient
//     and one residual correction (P. Markstein, "Computation of elementary
//     functions on the IBM RISC System/6000 processor", IBM J. R&D 34, 1990;
//     M. Cornea, J. Harrison, P. Tang, "Scientific Computing on Itanium-based
//     Systems", 2002): with the reciprocal correctly rounded the corrected
//     quotient is the correctly rounded one.  The operands here are in range
//     by construction, so no special cases.
// Float: a function of one float can be compared on every float, and was:
// ldpc_probe_sp_math does it (2 x 1e9 values, no difference).  On that
// evidence two of the float steps are shorter than the theorem needs (no
// Newton step for s, no residual for the last correction term).  Double: every
// division takes the full form; compared on random and boundary arguments.
#pragma once
#include <stdint.h>

#include "ldpc_math.h"

namespace ldpc {

__device__ __forceinline__ float spm_rcp(float d) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return r;
}
__device__ __forceinline__ double spm_rcp(double d) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    return r;
}

// quotient n / d from a reciprocal r of d, corrected by its residual
__device__ __forceinline__ float spm_quot(float n, float d, float r) {
    const float q = __fmul_rn(n, r);
    return __fmaf_rn(__fmaf_rn(-d, q, n), r, q);
}
__device__ __forceinline__ double spm_quot(double n, double d, double r) {
    const double q = __dmul_rn(n, r);
    return __fma_rn(__fma_rn(-d, q, n), r, q);
}

// n / d rounded to nearest
__device__ __forceinline__ float spm_div(float n, float d) {
    float r = spm_rcp(d);
    r = __fmaf_rn(r, __fmaf_rn(-d, r, 1.0f), r);
    return spm_quot(n, d, r);
}
__device__ __forceinline__ double spm_div(double n, double d) {
    double r = spm_rcp(d);                              // ~20 bits
    const double e = __fma_rn(-d, r, 1.0);
    // ~60 bits, rounded up to 53: from above, the next step is correctly
    // rounded for the divisor with an all-ones mantissa too (from below it ties)
    r = __fma_ru(r, __fma_rn(e, e, e), r);
    r = __fma_rn(r, __fma_rn(-d, r, 1.0), r);
    return spm_quot(n, d, r);
}

// tanh(a / 2), a >= 0
__device__ __forceinline__ float spm_tanh_half(float a) {
    const bool small = a < 0.25f;
    const float km = __fadd_rn(__fmul_rn(a, 1.44269502162933349609375f), 12582912.0f);
    const float k = __fsub_rn(km, 12582912.0f);
    const float r = __fmaf_rn(k, 1.428606765330187045e-06f, __fmaf_rn(k, 0.693145751953125f, -a));
    const float v = small ? -a : r;
    float p = small ? 2.7557319223985891e-06f : 0.0f;   // 1/9!
    p = __fmaf_rn(p, v, 2.4801587301587302e-05f);
    p = __fmaf_rn(p, v, 1.9841269841269841e-04f);
    p = __fmaf_rn(p, v, 1.3888888888888889e-03f);
    p = __fmaf_rn(p, v, 8.3333333333333333e-03f);
    p = __fmaf_rn(p, v, 4.1666666666666667e-02f);
    p = __fmaf_rn(p, v, 1.6666666666666667e-01f);
    p = __fmaf_rn(p, v, 0.5f);
    p = __fmaf_rn(p, v, 1.0f);
    const float scale = __int_as_float(0x3f800000 - (__float_as_int(km) << 23));   // 2^-k
    const float big = __fsub_rn(__fmul_rn(__fmaf_rn(p, v, 1.0f), scale), 1.0f);
    const float e = small ? __fmul_rn(p, v) : big;      // expm1(-a)
    const float q = spm_div(-e, __fadd_rn(2.0f, e));
    return a < 20.0f ? q : 1.0f;
}

// 2 atanh(m) = log1p(2 m / (1 - m)), 0 <= m <= 1
__device__ __forceinline__ float spm_atanh_twice(float m) {
    const float t = spm_div(__fadd_rn(m, m), __fsub_rn(1.0f, m));
    const bool small = t < 0.25f;
    const float u = __fadd_rn(1.0f, t);
    const int iu = __float_as_int(u);
    // exponent e of u = 2^e f, f in (1/sqrt 2, sqrt 2]: the mantissa of f > 1.41421356f carries
    const int eb = ((iu + (0x00800000 - 0x003504f4)) & 0x7f800000) - 0x3f800000;
    const float f = __int_as_float(iu - eb);
    const float e = __fsub_rn(__int_as_float((eb >> 23) + 0x4b000000), 8388608.0f);
    const float num = small ? t : __fsub_rn(f, 1.0f);
    const float den = small ? __fadd_rn(2.0f, t) : __fadd_rn(f, 1.0f);
    const float s = spm_quot(num, den, spm_rcp(den));
    const float s2 = __fmul_rn(s, s);
    float p = 7.6923076923076923e-02f;                  // 1/13
    p = __fmaf_rn(p, s2, 9.0909090909090909e-02f);
    p = __fmaf_rn(p, s2, 1.1111111111111111e-01f);
    p = __fmaf_rn(p, s2, 1.4285714285714286e-01f);
    p = __fmaf_rn(p, s2, 2.0000000000000000e-01f);
    p = __fmaf_rn(p, s2, 3.3333333333333333e-01f);
    p = __fmaf_rn(p, s2, 1.0f);
    const float ls = __fmul_rn(2.0f, __fmul_rn(p, s));
    const float corr = __fmul_rn(__fsub_rn(t, __fsub_rn(u, 1.0f)), spm_rcp(u));
    const float lo = __fadd_rn(__fmaf_rn(e, 1.428606765330187045e-06f, ls), corr);
    return small ? ls : __fmaf_rn(e, 0.693145751953125f, lo);
}

__device__ __forceinline__ double spm_tanh_half(double a) {
    const bool small = a < 0.25;
    const double km = __dadd_rn(__dmul_rn(a, 1.4426950408889634), 6755399441055744.0);
    const double k = __dsub_rn(km, 6755399441055744.0);
    const double r = __fma_rn(k, LMD_LN2_LO, __fma_rn(k, LMD_LN2_HI, -a));
    const double v = small ? -a : r;
    double p = 1.1470745597729725e-11;                  // 1/14!
    p = __fma_rn(p, v, 1.6059043836821613e-10);
    p = __fma_rn(p, v, 2.08767569878681e-09);
    p = __fma_rn(p, v, 2.505210838544172e-08);
    p = __fma_rn(p, v, 2.7557319223985888e-07);
    p = __fma_rn(p, v, 2.7557319223985893e-06);
    p = __fma_rn(p, v, 2.4801587301587302e-05);
    p = __fma_rn(p, v, 1.9841269841269841e-04);
    p = __fma_rn(p, v, 1.3888888888888889e-03);
    p = __fma_rn(p, v, 8.3333333333333332e-03);
    p = __fma_rn(p, v, 4.1666666666666664e-02);
    p = __fma_rn(p, v, 1.6666666666666666e-01);
    p = __fma_rn(p, v, 0.5);
    p = __fma_rn(p, v, 1.0);
    const double scale = __hiloint2double(0x3ff00000 - (__double2loint(km) << 20), 0);   // 2^-k
    const double big = __dsub_rn(__dmul_rn(__fma_rn(p, v, 1.0), scale), 1.0);
    const double e = small ? __dmul_rn(p, v) : big;     // expm1(-a)
    const double q = spm_div(-e, __dadd_rn(2.0, e));
    return a < 40.0 ? q : 1.0;
}

__device__ __forceinline__ double spm_atanh_twice(double m) {
    const double t = spm_div(__dadd_rn(m, m), __dsub_rn(1.0, m));
    const bool small = t < 0.25;
    const double u = __dadd_rn(1.0, t);
    const int hu = __double2hiint(u), lu = __double2loint(u);
    // f > 1.4142135623730951 (mantissa 0x6a09e 667f3bcd) goes to the next exponent
    const int up = (hu & 0xfffff) > 0x6a09e || ((hu & 0xfffff) == 0x6a09e && (uint32_t)lu > 0x667f3bcdu);
    const int ei = ((hu >> 20) & 0x7ff) - 1023 + up;
    const double f = __hiloint2double(hu - (ei << 20), lu);
    const double e = __dsub_rn(__hiloint2double(0x43380000, ei), 6755399441055744.0);
    const double num = small ? t : __dsub_rn(f, 1.0);
    const double den = small ? __dadd_rn(2.0, t) : __dadd_rn(f, 1.0);
    const double s = spm_div(num, den);
    const double s2 = __dmul_rn(s, s);
    double p = 0.040000000000000001;                    // 1/25
    p = __fma_rn(p, s2, 0.043478260869565216);
    p = __fma_rn(p, s2, 0.047619047619047616);
    p = __fma_rn(p, s2, 0.052631578947368418);
    p = __fma_rn(p, s2, 0.058823529411764705);
    p = __fma_rn(p, s2, 0.066666666666666666);
    p = __fma_rn(p, s2, 0.076923076923076927);
    p = __fma_rn(p, s2, 0.090909090909090912);
    p = __fma_rn(p, s2, 0.1111111111111111);
    p = __fma_rn(p, s2, 0.14285714285714285);
    p = __fma_rn(p, s2, 0.20000000000000001);
    p = __fma_rn(p, s2, 0.33333333333333331);
    p = __fma_rn(p, s2, 1.0);
    const double ls = __dmul_rn(2.0, __dmul_rn(p, s));
    const double corr = spm_div(__dsub_rn(t, __dsub_rn(u, 1.0)), u);
    const double lo = __dadd_rn(__fma_rn(e, LMD_LN2_LO, ls), corr);
    const double big = __fma_rn(e, LMD_LN2_HI, lo);
    return small ? ls : m < 1.0 ? big : __longlong_as_double((long long)0xfff8000000000000ull);
}

}  // namespace ldpc
