// Double-precision division and square root, correctly rounded, on the integer and FP32 pipes.
//
// GB300 issues one FP64 warp instruction per SM every 16 clocks but 4 integer or FP32 ones every clock, and the
// library's __ddiv_rn and __dsqrt_rn are chains of about ten FP64 instructions.  The functions here take about 60
// integer and FP32 instructions and no FP64 one: a float estimate gives the first ~20 bits of the quotient (or root),
// and two more digits follow from exact 64-bit remainders -- long division in base 2^20 with float digit estimates.
// The estimates are biased low, so each remainder and digit is non-negative, and the last remainder decides the
// rounding exactly: neither a quotient nor a root of doubles can lie halfway between two doubles.  So the values are
// __ddiv_rn's and __dsqrt_rn's bit for bit; operands or results outside the range the digits cover (zeros,
// subnormals, infinities, NaN, exponents within 2 of the limits) take those functions.
//
// Measured with atan2_int below (before -> after, one GB300): the mesh functions' exact form, 261,632 queries x 102
// segments, 5.84 -> 3.57 ms; the robust evaluator's under int64_grid, 150,000 queries on two tori with 6
// holes (41 to 87 segments with the seed), 2.52 -> 1.01 ms.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#include <cuda_runtime.h>

#include "approx.cuh"
#define AGWN_FN __device__ __forceinline__
#define AGWN_TABLE static __device__ const
#else // a host build of the same functions, for the tests
#define AGWN_FN inline
#define AGWN_TABLE static const
#endif

namespace agwn
{
#ifdef __CUDACC__
__device__ __forceinline__ uint64_t bits_of(double a)
{
    return uint64_t(__double_as_longlong(a));
}
__device__ __forceinline__ double of_bits(uint64_t b)
{
    return __longlong_as_double((long long)(b));
}
__device__ __forceinline__ float float_of_bits(uint32_t b)
{
    return __uint_as_float(b);
}
__device__ __forceinline__ uint32_t bits_of_float(float f)
{
    return __float_as_uint(f);
}
// out of line: the cases they serve are rare, and their registers and FP64 instructions stay out of the callers
// (inlined, the multiplication would be issued for every operand and then selected)
static __device__ __noinline__ double mul_general(double a, double b)
{
    return __dmul_rn(a, b);
}
static __device__ __noinline__ double div_general(double a, double b)
{
    return __ddiv_rn(a, b);
}
static __device__ __noinline__ double sqrt_general(double a)
{
    return __dsqrt_rn(a);
}
static __device__ __noinline__ double atan2_general(double y, double x)
{
    return atan2(y, x);
}
#else
template <class To, class From>
inline To copy_bits(From f)
{
    To t;
    static_assert(sizeof(To) == sizeof(From), "same size");
    std::memcpy(&t, &f, sizeof(t));
    return t;
}
inline uint64_t bits_of(double a)
{
    return copy_bits<uint64_t>(a);
}
inline double of_bits(uint64_t b)
{
    return copy_bits<double>(b);
}
inline float float_of_bits(uint32_t b)
{
    return copy_bits<float>(b);
}
inline uint32_t bits_of_float(float f)
{
    return copy_bits<uint32_t>(f);
}
inline double mul_general(double a, double b)
{
    return a * b;
}
inline double div_general(double a, double b)
{
    return a / b;
}
inline double sqrt_general(double a)
{
    return std::sqrt(a);
}
inline double atan2_general(double y, double x)
{
    return std::atan2(y, x);
}
// AGWN_APPROX_ERROR(): a relative error to add, so that a test covers the hardware's approximations
#ifndef AGWN_APPROX_ERROR
#define AGWN_APPROX_ERROR() 0.0
#endif
inline float rcp_approx(float x)
{
    return float((1.0 + (AGWN_APPROX_ERROR())) / x);
}
inline float rsqrt_approx(float x)
{
    return float((1.0 + (AGWN_APPROX_ERROR())) / std::sqrt(double(x)));
}
#endif

// The top 24 bits of a double's significand (high word h, low word l) as a float in [1, 2).
AGWN_FN float lead_float(uint32_t h, uint32_t l)
{
    return float_of_bits((((h << 3) | (l >> 29)) & 0x007fffffu) | 0x3f800000u);
}

// Integers as doubles by their bits, exact: |v| < 2^32, and |v| < 2^53.  (The conversion instructions run at the FP64
// rate.)
AGWN_FN uint32_t leading_zeros(uint32_t v)
{
#ifdef __CUDACC__
    return uint32_t(__clz(int(v)));
#else
    return v ? uint32_t(__builtin_clz(v)) : 32u;
#endif
}
AGWN_FN double double_of(int32_t v)
{
    uint32_t const m = v < 0 ? 0u - uint32_t(v) : uint32_t(v), z = leading_zeros(m);
    uint32_t const t = z < 32 ? m << z : 0u; // the leading one at bit 31
    uint32_t const h = (t >> 11) + ((1053u - z) << 20) + (uint32_t(v) & 0x80000000u);
    return of_bits(m ? (uint64_t(h) << 32) | (t << 21) : 0ull);
}
AGWN_FN double double_of_53(int64_t v)
{
    uint64_t const m = v < 0 ? 0ull - uint64_t(v) : uint64_t(v);
    uint32_t const h = uint32_t(m >> 32), z = h ? leading_zeros(h) : 32 + leading_zeros(uint32_t(m));
    uint64_t const t = m << (z & 63u); // the leading one at bit 63
    return of_bits(m ? (t >> 11) + (uint64_t(1085u - z) << 52) + (uint64_t(v) & 0x8000000000000000ull) : 0ull);
}

// a b, rounded to nearest even: the significands' 128-bit product by 32-bit halves, for operands within 2^+-511 (so
// the product is normal); the FP64 instruction for the others.  Some 40 integer instructions, which leave the FP64
// pipe to the sums: the mesh functions' exact form (27 products and 38 other FP64 instructions per term) went from 3.53
// to 2.25 ms on 261,632 queries x 102 segments, FP64 75% and integer pipe 62% busy.  For kernels with warps enough to
// hide its longer chain, and few enough copies for the instruction cache.
AGWN_FN double mul_rn_int(double a, double b)
{
    uint64_t const ab = bits_of(a), bb = bits_of(b);
    uint32_t const ah = uint32_t(ab >> 32), bh = uint32_t(bb >> 32), al = uint32_t(ab), bl = uint32_t(bb);
    if (2 * ah - (512u << 21) >= (1023u << 21) || 2 * bh - (512u << 21) >= (1023u << 21))
        return mul_general(a, b);
    // significands in [2^63, 2^64)
    uint32_t const a1 = (ah << 11) | (al >> 21) | 0x80000000u, a0 = al << 11;
    uint32_t const b1 = (bh << 11) | (bl >> 21) | 0x80000000u, b0 = bl << 11;
    uint64_t const ll = uint64_t(a0) * b0;
    uint64_t const m1 = uint64_t(a1) * b0 + (ll >> 32);
    uint64_t const m2 = uint64_t(a0) * b1 + uint32_t(m1);
    uint64_t h = uint64_t(a1) * b1 + (m1 >> 32) + (m2 >> 32);
    uint32_t const sticky = (uint32_t(m2) | uint32_t(ll)) ? 1u : 0u;
    uint32_t const top = uint32_t(h >> 63); // 0: the product is below 2^127, one bit less
    h = top ? h : h + h;
    uint64_t const M = h >> 11;
    uint32_t const rest = (uint32_t(h) & 0x7ffu) | sticky; // half is 0x400
    uint32_t const up = rest + (uint32_t(M) & 1u) > 0x400u ? 1u : 0u;
    uint32_t const e = (ah & 0x7ff00000u) + (bh & 0x7ff00000u) - ((1024u - top) << 20);
    return of_bits((uint64_t(e | ((ah ^ bh) & 0x80000000u)) << 32) + M + up);
}

// a / b, rounded to nearest even.
//
// With A, B the 53-bit significands, the quotient A / B in (1/2, 2) is built in units of 2^-55 as
// D0 2^34 + D1 2^15 + D2.  D0 is the float quotient less 2^-18 in units of 2^-21 (relative error below 2^-20, so the
// rest e0 = A/B - D0 2^-21 lies in (0, 2^-17)), D1 the float quotient of the first remainder less its own error bound
// in units of 2^-40 (below 2^23; the rest is in (0, 2^-35)), D2 the rounded float quotient of the second (below
// 2^20 + 1).  The third remainder, at most 0.6 B in magnitude, tells on which side of Q the quotient lies.
AGWN_FN double div_normal(double a, double b) // normal operands, e = exponent(a) - exponent(b) + 1023 in [3, 2042]
{
    uint64_t const ab = bits_of(a), bb = bits_of(b);
    uint32_t const ah = uint32_t(ab >> 32), bh = uint32_t(bb >> 32);
    int const e = int((ah >> 20) & 0x7ffu) - int((bh >> 20) & 0x7ffu) + 1023;
    uint64_t const A = (ab & 0x000fffffffffffffull) | 0x0010000000000000ull;
    uint64_t const B = (bb & 0x000fffffffffffffull) | 0x0010000000000000ull;
    float const r = rcp_approx(lead_float(bh, uint32_t(bb)));
    float const t0 = std::fma(lead_float(ah, uint32_t(ab)), r, 3.99999618530273438f); // 4 - 2^-18: in [4.49, 6), units 2^-21
    uint32_t const D0 = bits_of_float(t0) - 0x40800000u;
    uint64_t const R0 = (A << 21) - uint64_t(D0) * B; // units 2^-21 of B: below 2^4 B
    // digit 1: R0 / B in units of 2^-19 of the ones above, R0 >> 26 below 2^31
    float const f1 = float(uint32_t(R0 >> 26));
    float const t1 = std::fma(f1, r * 0.0078125f, 8388600.f); // 2^26 2^19 2^-52 = 2^-7; 2^23 - 8
    uint32_t const D1 = bits_of_float(t1) - 0x4b000000u;
    uint64_t const R1 = (R0 << 19) - uint64_t(D1) * B;
    float const f2 = float(uint32_t(R1 >> 26));
    float const t2 = std::fma(f2, r * 0.00048828125f, 8388608.f); // 2^26 2^15 2^-52 = 2^-11
    uint32_t const D2 = bits_of_float(t2) - 0x4b000000u;
    int64_t const R2 = int64_t((R1 << 15) - uint64_t(D2) * B);
    uint64_t const Q = (uint64_t(D0) << 34) + (uint64_t(D1) << 15) + D2;
    // 53 bits: drop 3 bits of a quotient of 1 or more, 2 of one below, with the remainder's sign as a last bit
    int const s = 2 + int(Q >> 55);
    uint64_t const V = 2 * Q + uint64_t(int64_t(R2 >= 0 ? 1 : -1));
    uint64_t const M = (V + (1ull << s)) >> (s + 1);
    return of_bits((uint64_t((ah ^ bh) & 0x80000000u) << 32) + (uint64_t(uint32_t(e + s - 4)) << 52) + M);
}

AGWN_FN double div_rn_int(double a, double b)
{
    int const ea = int((bits_of(a) >> 52) & 0x7ffu), eb = int((bits_of(b) >> 52) & 0x7ffu);
    // normal operands and a normal quotient (its biased exponent is ea - eb + 1023 or one less)
    if (unsigned(ea - 1) >= 2046u || unsigned(eb - 1) >= 2046u || unsigned(ea - eb + 1020) >= 2040u)
        return div_general(a, b);
    return div_normal(a, b);
}

// sqrt(a), rounded to nearest even.
//
// a = A 2^(2k) with A in [1, 4): the root in [1, 2) is built in units of 2^-55 as D0 2^34 + D1 2^15 + D2, D0 from the
// float root less 2^-18, D1 and D2 from the remainders A - S^2 times half the float reciprocal root, D1 less its
// error bound.  The last remainder, A - S^2 in units of 2^-110, is exact modulo 2^64 and below 2^57 in magnitude.
AGWN_FN double sqrt_rn_int(double a)
{
    uint64_t const ab = bits_of(a);
    uint32_t const ah = uint32_t(ab >> 32);
    if (unsigned((ah >> 20) - 1) >= 2046u) // zero, subnormal, infinite, NaN or negative
        return sqrt_general(a);
    uint32_t const odd = (~ah >> 20) & 1u; // odd exponent (the bias is odd)
    uint64_t const X = ((ab & 0x000fffffffffffffull) | 0x0010000000000000ull) << odd; // A in units of 2^-52
    float const f = float_of_bits(bits_of_float(lead_float(ah, uint32_t(ab))) + (odd << 23));
    float const r = rsqrt_approx(f);
    float const t0 = std::fma(f, r, 3.99999618530273438f);
    uint32_t const D0 = bits_of_float(t0) - 0x40800000u; // root less up to 2^-17, units 2^-21
    uint64_t const R0 = X - (uint64_t(D0) * D0 << 10);   // units 2^-52: below 2^37
    float const f1 = float(uint32_t(R0 >> 6));
    float const t1 = std::fma(f1, r * 0.0078125f, 8388600.f); // R0 r / 2 in units of 2^-40: 2^6 2^-52 2^40 / 2 = 2^-7; 2^23 - 8
    uint32_t const D1 = bits_of_float(t1) - 0x4b000000u;
    uint64_t const S1 = (uint64_t(D0) << 19) + D1; // units 2^-40
    uint64_t const R1 = (X << 28) - S1 * S1;       // units 2^-80, below 2^48
    float const f2 = float(uint32_t(R1 >> 17));
    float const t2 = std::fma(f2, r * 0.001953125f, 8388608.f); // 2^17 2^-80 2^55 / 2 = 2^-9
    uint32_t const D2 = bits_of_float(t2) - 0x4b000000u;
    uint64_t const S2 = (S1 << 15) + D2; // units 2^-55
    int64_t const R2 = int64_t((X << 58) - S2 * S2);
    uint64_t const V = 2 * S2 + uint64_t(int64_t(R2 >= 0 ? 1 : -1));
    uint64_t const M = (V + 8) >> 4; // 53 bits, the leading one included
    uint32_t const e = ((ah >> 20) + 1021u) >> 1; // floor((field - 1023) / 2) + 1022: M carries the leading one
    return of_bits((uint64_t(e) << 52) + M);
}

// Entry 4 k + o: a double c within 2^-20 of k / 64 and the nearest double to atan(c), pi/2 - atan(c), pi - atan(c) or
// pi/2 + atan(c) (o = 0..3).  Each c is chosen (Gal's accurate tables) so that the angle lies within 2^-10 of an ulp of
// that double; tests/test_intfp.py checks the entries.
struct alignas(16) AtanEntry
{
    double c, angle;
};
AGWN_TABLE AtanEntry kAtanTable[260] = {
    {0.0, 0.0}, {8.642822451668009e-07, 1.5707954625126515},
    {5.171837404013407e-07, 3.141592136406053}, {4.474023719779933e-07, 1.5707967741972686},
    {0.01562504428966681, 0.015623772899333341}, {0.015624628574239964, 1.555172969509524},
    {0.015624680900949489, 3.1259692439904825}, {0.015624939849773875, 1.5864199952798288},
    {0.0312505214865098, 0.03124035440800227}, {0.031249072180063665, 1.5395574202794013},
    {0.031249677254695424, 3.1103531425899593}, {0.0312509103864205, 1.6020370697233777},
    {0.04687557705770137, 0.04684128870848635}, {0.04687508802343031, 1.5239555260484838},
    {0.04687573216703202, 3.094751210112055}, {0.046874540228478624, 1.6176365809473603},
    {0.0625007812183115, 0.06241958817447103}, {0.0625003688723201, 1.5083771493619285},
    {0.06249949836881142, 3.0791743432731677}, {0.06250039706386579, 1.6332155323097144},
    {0.07812431106903164, 0.07796594907992926}, {0.07812416953788326, 1.4928305183875352},
    {0.07812419079527246, 3.0636268240539977}, {0.07812559237997321, 1.6487635494127186},
    {0.0937491687127395, 0.0934759571138455}, {0.093749192983229, 1.4773203456220143},
    {0.09374937713506527, 3.048116489869471}, {0.0937507370088054, 1.6642738385410611},
    {0.10937560689616792, 0.10894255671158853}, {0.10937471351243226, 1.4618546529059027},
    {0.1093754647250088, 3.0326502373686752}, {0.109374190230631, 1.679737483587989},
    {0.12499970639586173, 0.12435470545959947}, {0.1250002623720543, 1.4464410739125824},
    {0.12499979893056898, 3.017237857019092}, {0.12499959887457672, 1.6951509263873756},
    {0.1406252135499747, 0.1397090836979907}, {0.1406243822183117, 1.4310880583075072},
    {0.1406251623070257, 3.0018836201410504}, {0.1406248760017548, 1.7105050794903756},
    {0.15625027495639837, 0.1549970103275064}, {0.15624940088159928, 1.4158001697110876},
    {0.15625049734482352, 2.9865954261738974}, {0.15624906988337273, 1.7257921607688267},
    {0.1718758502882541, 0.17021275117596396}, {0.17187541301597975, 1.4005840003442962},
    {0.171875152359502, 2.9713805803165303}, {0.17187489074893966, 1.7410081459640914},
    {0.18750071617967942, 0.18534864185220098}, {0.18750021043894058, 1.385448173507252},
    {0.18750067126763806, 2.956244055124308}, {0.18750041482856444, 1.7561446775306084},
    {0.20312463459197622, 0.2003982028970691}, {0.2031254139731977, 1.3703973753994798},
    {0.20312430844705148, 2.9411947639142686}, {0.20312562056124442, 1.771195476592299},
    {0.2187502784810711, 0.21535796546157795}, {0.21875024386011785, 1.3554383943732555},
    {0.21875071552141476, 2.926234271045998}, {0.21875068346286353, 1.7861546787441467},
    {0.23437433110864445, 0.23021895321542288}, {0.23437436802803752, 1.3405773385825106},
    {0.2343757601162777, 2.911372345777021}, {0.2343745927444835, 1.8010155280225049},
    {0.24999953491052976, 0.24497822539555014}, {0.25000046826865385, 1.325817222944642},
    {0.2499995113122622, 2.8966144504043823}, {0.2499996932730586, 1.8157747012375598},
    {0.2656245994802299, 0.2596292552853062}, {0.2656257320858601, 1.3111660135501195},
    {0.26562443784993833, 2.881963549282328}, {0.26562499546586116, 1.8304259519678445},
    {0.2812498251488758, 0.27416728908566845}, {0.2812505366052645, 1.2966283784049084},
    {0.28125019128586703, 2.867425025206136}, {0.2812492797983319, 1.8449631105058255},
    {0.29687529138840985, 0.2885876296811162}, {0.2968743184786529, 1.2822095912216531},
    {0.2968745822723107, 2.8530056755890993}, {0.2968756307780252, 1.8593842683762853},
    {0.31250075787560955, 0.3028855588237763}, {0.3124993790686551, 1.267912024108368},
    {0.31250019861633416, 2.8387076042689903}, {0.31249976487888387, 1.8736809809669863},
    {0.3281258241367221, 0.31705649723894413}, {0.3281251696997596, 1.253740420380949},
    {0.3281257565458079, 2.8245362173718442}, {0.3281250639737369, 1.8878521377594815},
    {0.3437492261490101, 0.3310953846311171}, {0.34374973094849043, 1.2397004907097764},
    {0.3437494204236976, 2.8104970952142545}, {0.3437492310703859, 1.901891715827316},
    {0.35937529094527443, 0.345002434874507}, {0.35937587451587666, 1.2257933750978383},
    {0.35937427069162525, 2.7965911222741036}, {0.3593750298343783, 1.915798530423972},
    {0.3749993791778281, 0.35877012598800906}, {0.3750001921309422, 1.2120254880807693},
    {0.375000558403723, 2.7828214937598825}, {0.37499965093538723, 1.9295666910361842},
    {0.3906253088438257, 0.37239871463358065}, {0.39062405398661776, 1.1983987008917192},
    {0.39062517399330415, 2.769194055954231}, {0.390624344874211, 1.9431942050760085},
    {0.4062499134271547, 0.38588259508910794}, {0.4062496925951266, 1.184913921254848},
    {0.40624986212776626, 2.755710102533022}, {0.40624910616009724, 1.9566782289739044},
    {0.421874388440885, 0.3992202504153181}, {0.42187469012030276, 1.171575820280241},
    {0.4218750146908211, 2.7423718715433276}, {0.4218744640942019, 1.9700166414332434},
    {0.43749950346947913, 0.4124100248372676}, {0.4375004763458062, 1.15838548537946},
    {0.43749958174287096, 2.7291825630541813}, {0.4374998968589951, 1.98320668182147},
    {0.4531257680728659, 0.42545027460430407}, {0.4531252549744315, 1.1453464778844105},
    {0.4531256742500333, 2.716142456825901}, {0.45312503014293726, 1.9962459891731361},
    {0.46874943708199296, 0.4383360983462173}, {0.46874912052790363, 1.1324604879775562},
    {0.4687506255259816, 2.7032555808908016}, {0.4687500366280531, 2.009132916682579},
    {0.4843755123581626, 0.45107007098132795}, {0.4843756754812083, 1.119726123689447},
    {0.48437557674503406, 2.690522530457286}, {0.48437497986679956, 2.0218659664762044},
    {0.49999915328384936, 0.4636469316276562}, {0.4999992387375257, 1.1071493268042554},
    {0.4999991072888992, 2.677945758758123}, {0.5000001261348056, 2.034444036703542},
    {0.5156243182654843, 0.47606879177206657}, {0.5156242048892297, 1.0947276245868451},
    {0.5156258982746582, 2.6655226136562984}, {0.5156258789992196, 2.0468663515013636},
    {0.531250360509575, 0.4883342322153923}, {0.5312503691653314, 1.0824620878289393},
    {0.5312491633472249, 2.6532593550335695}, {0.5312494945015662, 2.0591298836163405},
    {0.5468743125642749, 0.5004402839727884}, {0.5468746473173233, 1.0703557851357548},
    {0.5468758624457033, 2.641151176549186}, {0.54687577191341, 2.0712377341455923},
    {0.5624991054072715, 0.5123887807385537}, {0.5624997728667583, 1.058407039024561},
    {0.5625007297335445, 2.6292026389415804}, {0.5625006906566046, 2.083186311758568},
    {0.5781253442785774, 0.5241798868185661}, {0.5781257380886753, 1.0466161448170617},
    {0.5781258188990009, 2.617412411044919}, {0.5781243357623285, 2.094975457733659},
    {0.5937492893590663, 0.5358107125477972}, {0.5937501257767902, 1.0349849958413455},
    {0.5937491134920517, 2.605782071069396}, {0.5937498027457637, 2.1066074189153925},
    {0.6093758670786412, 0.5472850132738436}, {0.6093741117948622, 1.0235125935001212},
    {0.6093752589950107, 2.5943080837393615}, {0.6093754243132966, 2.1180810171978464},
    {0.6250009449971275, 0.55859999489177}, {0.625000265687421, 1.012196820395234},
    {0.6249991275701389, 2.58299396561177}, {0.6250004132665974, 2.1293959393188784},
    {0.6406244607920515, 0.5697560711744623}, {0.6406255685457518, 1.0010394702025538},
    {0.6406244407881686, 2.5718365965984615}, {0.6406244306125705, 2.140552376571537},
    {0.6562492854082379, 0.5807558540849371}, {0.6562497792428437, 0.9900401275312201},
    {0.656250898857423, 2.5608356717425176}, {0.6562501986390415, 2.1515528192064988},
    {0.67187580738238, 0.5916002666071034}, {0.6718747307341073, 0.9791968019792526},
    {0.6718742137582674, 2.549993484961546}, {0.6718754923777224, 2.162396376369485},
    {0.6875000131888355, 0.6022873550907781}, {0.6874997037810004, 0.9685091818060183},
    {0.6875006448596513, 2.539304869566179}, {0.6875005297254829, 2.1730840326372616},
    {0.703124586734769, 0.6128199256197887}, {0.7031251522659174, 0.9579760227376192},
    {0.7031247784444711, 2.528772599683258}, {0.7031254714186718, 2.183616844420104},
    {0.7187494929447478, 0.6231989955974896}, {0.7187496010262652, 0.9475972599317783},
    {0.7187496255198147, 2.5183935705763827}, {0.718750306059962, 2.193995858535373},
    {0.7343745645604902, 0.6334256000887952}, {0.7343754222224337, 0.9373701695318996},
    {0.7343742680052193, 2.508167246156203}, {0.7343741322617091, 2.2042216460435795},
    {0.7499994237006063, 0.6435007399615704}, {0.7500007029869304, 0.9272947680901286},
    {0.7500007421906832, 2.498091069794641}, {0.7500005596524454, 2.21429779376565},
    {0.7656256654062691, 0.6534267606825632}, {0.7656241367685257, 0.9173705298341734},
    {0.7656247336333557, 2.488166480338524}, {0.7656245905085558, 2.2242224098138474},
    {0.7812497607801174, 0.663202844154736}, {0.7812508733579643, 0.9075927917490966},
    {0.7812498375784015, 2.478389761744664}, {0.7812499207569483, 2.2339992702924465},
    {0.7968742041258001, 0.6728320608232708}, {0.7968752230212037, 0.897963642797557},
    {0.796875766338748, 2.4687596372902902}, {0.7968755302326681, 2.243629198687965},
    {0.8125005639906719, 0.6823168945960943}, {0.8125004321702557, 0.888479511601179},
    {0.8125003947170528, 2.4592758609561134}, {0.812500695561282, 2.253113300642886},
    {0.8281257569746147, 0.6916570708853315}, {0.82812414702103, 0.8791402109233514},
    {0.828125374428352, 2.44993580962823}, {0.8281252530915008, 2.26245309878027},
    {0.8437504373952973, 0.7008546633851278}, {0.8437493886541724, 0.8699422760230056},
    {0.8437505478484509, 2.440737925684429}, {0.843750565254089, 2.2716510648676103},
    {0.8593744016868141, 0.7099112743136113}, {0.8593754773914465, 0.8608844337358229},
    {0.8593751598021105, 2.4316809432080837}, {0.8593750488829205, 2.280707973375882},
    {0.8749994193082085, 0.7188296707341435}, {0.8749994197429706, 0.851966655814516},
    {0.8749992917803657, 2.4227630550838546}, {0.8750005219243439, 2.289626622019613},
    {0.8906248479231389, 0.7276112478195849}, {0.8906248797957343, 0.8431850612012929},
    {0.8906250726709218, 2.4139812804377434}, {0.8906248614631559, 2.298407582165185},
    {0.906250215007402, 0.736257547033737}, {0.9062492693753745, 0.8345392989715856},
    {0.9062500636422867, 2.4053351896648265}, {0.9062507612800165, 2.3070541737658377},
    {0.9218745210219527, 0.7447698667884587}, {0.921875464974919, 0.8260259497211829},
    {0.9218754461098212, 2.3968222867142326}, {0.9218756065616217, 2.3155667804079827},
    {0.9374996049453689, 0.7531510707043867}, {0.9375006026501603, 0.817644725087599},
    {0.9374993384541463, 2.3884417247186476}, {0.9374992656114427, 2.3239472168973414},
    {0.9531254655885816, 0.7614030137675059}, {0.9531246434615558, 0.8093937438105703},
    {0.9531250058638687, 2.3801898807116286}, {0.9531250128447586, 2.332199103330951},
    {0.9687508417133845, 0.7695269146193324}, {0.9687495856904031, 0.8012700601187673},
    {0.9687505056038401, 2.3720659123588446}, {0.968749998397383, 2.3403228063738144},
    {0.9843757182950946, 0.7775246751762803}, {0.984375232247763, 0.7932718984690719},
    {0.9843757501052443, 2.364067962257992}, {0.9843756546870711, 2.348320969666368},
    {0.9999995065598519, 0.7853979166773134}, {0.9999992247888422, 0.7853985510031775},
    {0.9999998583615368, 2.3561945610115815}, {0.9999994101968716, 2.3561941952906937}};
AGWN_FN AtanEntry atan_entry(uint32_t i)
{
#ifdef __CUDACC__
    double2 const e = __ldg(reinterpret_cast<const double2*>(kAtanTable) + i);
    return {e.x, e.y};
#else
    return kAtanTable[i];
#endif
}

// atan2(y, x) in double precision in 7 FP64 instructions (the library's takes about 35).  Errors in ulp over 1.5e6
// arguments each, mean and largest, the library's in brackets: the circle 0.106, 0.99 (0.151, 1.59); angles up to 0.05
// 0.279, 1.19 (0.339, 1.39); from 1/128 to 3/64 0.285, 1.13 (0.336, 1.46).
//
// With n <= d the smaller and larger of |y| and |x| and c the table's value next to n / d (from a float quotient), the
// addition formula gives atan(n / d) = atan(c) + atan(q), q = (n - c d) / (d + c n), |q| <= 2^-6.9.  Up to 3/256 c is 0 (or
// within 2^-20 of it) in place of 1/64: q is then one rounded quotient, where the difference to 1/64 would be as large as
// the angle with three roundings in it.  Both terms of q are one FMA, the quotient is div_normal's, and atan(q) = q - q^3/3
// + q^5/5 - q^7/7 + q^9/9 is cut below 2^-67 relative (2^-60 at 3/256).  The
// octant is folded into the table's angle, so one addition ends it.  Zeros and operands beyond 2^+-383 (subnormals,
// infinities, NaN) take the library's function.
AGWN_FN double atan2_int(double y, double x)
{
    uint64_t const yb = bits_of(y) & 0x7fffffffffffffffull, xb = bits_of(x) & 0x7fffffffffffffffull;
    bool const swap = yb > xb;
    uint64_t const nb = swap ? xb : yb, db = swap ? yb : xb;
    uint32_t const nh = uint32_t(nb >> 32), dh = uint32_t(db >> 32);
    int const en = int(nh >> 20), ed = int(dh >> 20);
    if (unsigned(en - 640) >= 768u || unsigned(ed - 640) >= 768u)
        return atan2_general(y, x);
    // n / d in float: both over 2^(exponent of d); below 2^-60 it is 0
    float const fd = lead_float(dh, uint32_t(db));
    float const fn = en < ed - 60 ? 0.f
                                  : float_of_bits(((nh - (uint32_t(ed) << 20) + (127u << 20)) << 3) |
                                                  (uint32_t(nb) >> 29));
    float const t64 = fn * (rcp_approx(fd) * 64.f);
    uint32_t const k = t64 < 0.75f ? 0u : bits_of_float(t64 + 8388608.f) & 0x7fu;
    double const n = of_bits(nb), d = of_bits(db);
    // the octant: bit 0 the swap, bit 1 x < 0
    uint32_t const neg = uint32_t(bits_of(x) >> 63), sw = swap ? 1u : 0u;
    AtanEntry const t = atan_entry(4 * k + 2 * neg + sw);
    double const num = std::fma(-t.c, d, n), den = std::fma(t.c, n, d);
    double q = div_normal(num, den);
    if ((bits_of(num) & 0x7ff0000000000000ull) == 0)
        q = 0.0;
    uint64_t const qb = bits_of(q);
    // 1/5 - q^2/7 + q^4/9 from q^2 in float (0 when q is below float's range): the difference to 1/5 in units of 2^-38
    // (below 2^23), off the significand of 1/5
    uint32_t const qh = uint32_t(qb >> 32) & 0x7fffffffu;
    float const qf = qh < (900u << 20) ? 0.f : float_of_bits((qh - (896u << 20)) << 3);
    float const s = qf * qf;
    float const t38 = std::fma(s, std::fma(s, -0x1.c71c72p+34f, 0x1.24924ap+35f), 8388608.f);
    double const inner = of_bits(0x3fc999999999999aull - (uint64_t(bits_of_float(t38) - 0x4b000000u) << 17));
    double const q2 = q * q;
    double const r = std::fma(q * q2, std::fma(q2, inner, -0.33333333333333333), q);
    // angle + r or angle - r: minus when exactly one of the swap and x < 0 holds
    double const a = t.angle + of_bits(bits_of(r) ^ (uint64_t(neg ^ sw) << 63));
    return of_bits(bits_of(a) ^ (bits_of(y) & 0x8000000000000000ull));
}
} // namespace agwn
