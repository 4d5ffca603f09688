// The double-float operators (csrc/df32.cuh) built for the host, beside plain ones: sums and products composed from the
// add and the multiply, the quotient from two residuals in double-float.  Prints, per operator, the mean and the largest
// error of the library's and of the plain one, over random operands and in extended precision; sums' errors relative to
// the sum of the magnitudes.  The approximate reciprocals carry a random error of up to 2^-22.9, the same for both.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <random>

static double approx_error = 0;
#define AGWN_APPROX_ERROR() approx_error
#include "../../antipodal_gb300/csrc/df32.cuh"

using namespace agwn;

static df plain_quotient(df a, df b)
{
    float const rb = rcp_approx(b.hi), q1 = a.hi * rb;
    df const r = a - b * df_make(q1);
    float const q2 = r.hi * rb;
    df const q = fast_two_sum(q1, q2), r2 = a - b * q;
    return q + df_make(r2.hi * rb);
}
static df plain_sqrt(df a)
{
    float const ri = rsqrt_approx(a.hi), y = a.hi * ri;
    df const e = a - two_prod(y, y);
    return fast_two_sum(y, e.hi * ri * 0.5f);
}

static std::mt19937_64 rng(1);
static double uniform()
{
    return double(rng() >> 11) * 0x1p-53;
}
static df operand(int spread)
{
    double const x = std::ldexp((rng() & 1 ? -1 : 1) * (1 + uniform()), int(rng() % (2 * spread + 1)) - spread);
    float const h = float(x);
    return fast_two_sum(h, float((uniform() - 0.5) * std::ldexp(1.0, std::ilogb(h) - 23)));
}
static long double value(df a)
{
    return (long double)(a.hi) + (long double)(a.lo);
}

struct Errors
{
    const char* name;
    double sum[2] = {0, 0}, most[2] = {0, 0};
    void add(df ours, df plain, long double exact, long double scale)
    {
        df const v[2] = {ours, plain};
        for (int k = 0; k < 2; ++k)
        {
            double const e = double(std::fabs((value(v[k]) - exact) / scale));
            sum[k] += e;
            most[k] = std::max(most[k], e);
        }
    }
};

int main()
{
    constexpr int n = 2000000;
    Errors quotient{"quotient"}, root{"root"}, fma{"fma"}, dot{"dot"}, det{"det"};
    for (int i = 0; i < n; ++i)
    {
        approx_error = 2.55e-7 * (uniform() - 0.5);
        df const a = operand(3), b = operand(3), c = operand(6), d = operand(3);
        long double const A = value(a), B = value(b), C = value(c), D = value(d);
        quotient.add(a / b, plain_quotient(a, b), A / B, A / B);
        df const r{std::fabs(a.hi), a.hi < 0 ? -a.lo : a.lo};
        root.add(df_sqrt(r), plain_sqrt(r), std::sqrt(value(r)), std::sqrt(value(r)));
        fma.add(df_fma(a, b, c), a * b + c, A * B + C, std::fabs(A * B) + std::fabs(C));
        dot.add(df_dot2(a, b, c, d), a * b + c * d, A * B + C * D, std::fabs(A * B) + std::fabs(C * D));
        det.add(df_det2(a, b, c, d), a * b - c * d, A * B - C * D, std::fabs(A * B) + std::fabs(C * D));
    }
    for (Errors const* e : {&quotient, &root, &fma, &dot, &det})
        std::printf("%s %.6e %.6e %.6e %.6e\n", e->name, e->sum[0] / n, e->most[0], e->sum[1] / n, e->most[1]);
    return 0;
}
