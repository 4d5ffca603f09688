// Double-float arithmetic: a value is hi + lo, two floats with |lo| <= ulp(hi) / 2, about 44 significant bits,
// computed on the FP32 pipe (64x the FP64 rate of this GPU).  Built from the error-free transformations TwoSum
// (Knuth), FastTwoSum (Dekker, |a| >= |b|) and TwoProduct by FMA; add is the "sloppy" variant (error relative to
// |a| + |b|), multiply folds the cross terms into the FMA error term, divide takes three float digits and sqrt one
// Newton-style correction of a float estimate.  Every step is written with explicit round-to-nearest intrinsics so
// the compiler cannot reassociate or contract them.
#pragma once

#include <cuda_runtime.h>

#include "approx.cuh"

namespace agwn
{
struct df
{
    float hi, lo;
};

__device__ __forceinline__ df df_from(double d)
{
    float const h = __double2float_rn(d);
    return {h, __double2float_rn(d - double(h))};
}
__device__ __forceinline__ double df_to(df a)
{
    return double(a.hi) + double(a.lo);
}
__device__ __forceinline__ df df_make(float hi)
{
    return {hi, 0.f};
}

__device__ __forceinline__ df fast_two_sum(float a, float b)
{
    float const s = __fadd_rn(a, b);
    return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ df two_sum(float a, float b)
{
    float const s = __fadd_rn(a, b);
    float const bb = __fsub_rn(s, a);
    return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
__device__ __forceinline__ df two_prod(float a, float b)
{
    float const p = __fmul_rn(a, b);
    return {p, __fmaf_rn(a, b, -p)};
}

__device__ __forceinline__ df df_neg(df a)
{
    return {-a.hi, -a.lo};
}
__device__ __forceinline__ df operator+(df a, df b)
{
    df const s = two_sum(a.hi, b.hi);
    return fast_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}
__device__ __forceinline__ df operator-(df a, df b)
{
    return a + df_neg(b);
}
__device__ __forceinline__ df operator*(df a, df b)
{
    df const p = two_prod(a.hi, b.hi);
    float const e = __fmaf_rn(a.lo, b.hi, __fmaf_rn(a.hi, b.lo, p.lo));
    return fast_two_sum(p.hi, e);
}
// exact scaling by a power of two
__device__ __forceinline__ df df_scale(df a, float p2)
{
    return {__fmul_rn(a.hi, p2), __fmul_rn(a.lo, p2)};
}
// a b + c in one chain: the product's two floats, its cross terms and c.lo go into one low word
__device__ __forceinline__ df df_fma(df a, df b, df c)
{
    df const p = two_prod(a.hi, b.hi);
    float const e = __fmaf_rn(a.lo, b.hi, __fmaf_rn(a.hi, b.lo, p.lo));
    df const s = two_sum(p.hi, c.hi);
    return fast_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(e, c.lo)));
}
// a b + c d, and a b - c d
__device__ __forceinline__ df df_dot2(df a, df b, df c, df d)
{
    df const p = two_prod(a.hi, b.hi), q = two_prod(c.hi, d.hi);
    float const e = __fmaf_rn(a.lo, b.hi, __fmaf_rn(a.hi, b.lo, p.lo));
    float const f = __fmaf_rn(c.lo, d.hi, __fmaf_rn(c.hi, d.lo, q.lo));
    df const s = two_sum(p.hi, q.hi);
    return fast_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(e, f)));
}
__device__ __forceinline__ df df_det2(df a, df b, df c, df d)
{
    return df_dot2(a, b, df{-c.hi, -c.lo}, d);
}
// a + b for |a| >= |b|
__device__ __forceinline__ df df_add_ordered(df a, df b)
{
    df const s = fast_two_sum(a.hi, b.hi);
    return fast_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}
// The quotient as three float digits q1 + q2 + q3 of one reciprocal; a.hi - q1 b.hi is exact in an FMA.
__device__ __forceinline__ df operator/(df a, df b)
{
    float const rb = rcp_approx(b.hi);
    float const q1 = __fmul_rn(a.hi, rb);
    float const r1 = __fmaf_rn(-q1, b.hi, a.hi), l = __fmaf_rn(-q1, b.lo, a.lo);
    float const q2 = __fmul_rn(__fadd_rn(r1, l), rb);
    float const r2 = __fadd_rn(__fmaf_rn(-q2, b.hi, r1), l);
    return fast_two_sum(q1, __fmaf_rn(r2, rb, q2));
}
__device__ __forceinline__ df df_sqrt(df a)
{
    if (!(a.hi > 0.f))
        return {sqrtf(a.hi), 0.f};
    float const ri = rsqrt_approx(a.hi);
    float const y = __fmul_rn(a.hi, ri);
    df const p = two_prod(y, y);
    float const e = __fadd_rn(__fsub_rn(__fsub_rn(a.hi, p.hi), p.lo), a.lo); // a.hi - p.hi is exact
    return fast_two_sum(y, __fmul_rn(__fmul_rn(e, ri), 0.5f));
}
} // namespace agwn
