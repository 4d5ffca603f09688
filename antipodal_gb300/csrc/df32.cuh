// Double-float arithmetic: a value is hi + lo, two floats with |lo| <= ulp(hi) / 2, about 44 significant bits,
// computed on the FP32 pipe (64x the FP64 rate of this GPU).  Built from the error-free transformations TwoSum
// (Knuth), FastTwoSum (Dekker, |a| >= |b|) and TwoProduct by FMA; add is the "sloppy" variant (error relative to
// |a| + |b|), multiply folds the cross terms into the FMA error term, divide takes three float digits and sqrt one
// Newton-style correction of a float estimate.  Every step is written with explicit round-to-nearest intrinsics so
// the compiler cannot reassociate or contract them (a host build, for the tests, wants -ffp-contract=off).
#pragma once

#include "intfp.cuh" // the approximate reciprocals

namespace agwn
{
#ifndef __CUDACC__
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
inline float __double2float_rn(double d) { return float(d); }
#endif
struct df
{
    float hi, lo;
};

AGWN_FN df df_from(double d)
{
    float const h = __double2float_rn(d);
    return {h, __double2float_rn(d - double(h))};
}
AGWN_FN double df_to(df a)
{
    return double(a.hi) + double(a.lo);
}
AGWN_FN df df_make(float hi)
{
    return {hi, 0.f};
}

AGWN_FN df fast_two_sum(float a, float b)
{
    float const s = __fadd_rn(a, b);
    return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
AGWN_FN df two_sum(float a, float b)
{
    float const s = __fadd_rn(a, b);
    float const bb = __fsub_rn(s, a);
    return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
AGWN_FN df two_prod(float a, float b)
{
    float const p = __fmul_rn(a, b);
    return {p, __fmaf_rn(a, b, -p)};
}

AGWN_FN df df_neg(df a)
{
    return {-a.hi, -a.lo};
}
AGWN_FN df operator+(df a, df b)
{
    df const s = two_sum(a.hi, b.hi);
    return fast_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}
AGWN_FN df operator-(df a, df b)
{
    return a + df_neg(b);
}
AGWN_FN df operator*(df a, df b)
{
    df const p = two_prod(a.hi, b.hi);
    float const e = __fmaf_rn(a.lo, b.hi, __fmaf_rn(a.hi, b.lo, p.lo));
    return fast_two_sum(p.hi, e);
}
// exact scaling by a power of two
AGWN_FN df df_scale(df a, float p2)
{
    return {__fmul_rn(a.hi, p2), __fmul_rn(a.lo, p2)};
}
// a b + c.  The product is normalised before the sum: three operations that hold the low word's rounding down (without
// them the largest error goes from 2^-46.1 to 2^-45.7 of |a b| + |c|).
AGWN_FN df df_fma(df a, df b, df c)
{
    return a * b + c;
}
// a b + c d, and a b - c d
AGWN_FN df df_dot2(df a, df b, df c, df d)
{
    return a * b + c * d;
}
AGWN_FN df df_det2(df a, df b, df c, df d)
{
    return df_dot2(a, b, df{-c.hi, -c.lo}, d);
}
// a + b for |a| >= |b|
AGWN_FN df df_add_ordered(df a, df b)
{
    df const s = fast_two_sum(a.hi, b.hi);
    return fast_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}
// The quotient as three float digits q1 + q2 + q3 of one reciprocal.  q1 is corrected once, to within an ulp of
// a.hi / b.hi, so that a.hi - q1 b.hi is exact in an FMA; q1 + q2 is normalised before q3 goes in.  Errors over 3e6 random
// operands: mean 2^-49.9, largest 2^-46.2 (two residuals a - b q in double-float: 2^-49.6 and 2^-46.1).
AGWN_FN df operator/(df a, df b)
{
    float const rb = rcp_approx(b.hi);
    float const q0 = __fmul_rn(a.hi, rb);
    float const q1 = __fmaf_rn(__fmaf_rn(-q0, b.hi, a.hi), rb, q0);
    float const r1 = __fmaf_rn(-q1, b.hi, a.hi), l = __fmaf_rn(-q1, b.lo, a.lo);
    float const q2 = __fmul_rn(__fadd_rn(r1, l), rb);
    float const r2 = __fmaf_rn(-q2, b.lo, __fadd_rn(__fmaf_rn(-q2, b.hi, r1), l));
    df const q = fast_two_sum(q1, q2);
    return fast_two_sum(q.hi, __fmaf_rn(r2, rb, q.lo));
}
AGWN_FN df df_sqrt(df a)
{
    if (!(a.hi > 0.f))
        return {std::sqrt(a.hi), 0.f};
    float const ri = rsqrt_approx(a.hi);
    float const y = __fmul_rn(a.hi, ri);
    df const p = two_prod(y, y);
    float const e = __fadd_rn(__fsub_rn(__fsub_rn(a.hi, p.hi), p.lo), a.lo); // a.hi - p.hi is exact
    return fast_two_sum(y, __fmul_rn(__fmul_rn(e, ri), 0.5f));
}
} // namespace agwn
