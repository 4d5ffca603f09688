// The integer-pipe division, square root, atan2 and product (csrc/intfp.cuh) built for the host: reads n pairs (a, b)
// from standard input as raw doubles and writes a / b, sqrt(a), atan2(a, b) and a b for each.  The float estimates carry a
// random relative error of up to 2^-22.4, as the hardware's approximate reciprocals do.
#include <cstdio>
#include <cstdlib>

static double approx_error()
{
    return 3.6e-7 * (std::rand() / (RAND_MAX + 1.0) - 0.5);
}
#define AGWN_APPROX_ERROR() approx_error()
#include "../../antipodal_gb300/csrc/intfp.cuh"

int main()
{
    double in[2];
    while (std::fread(in, sizeof(double), 2, stdin) == 2)
    {
        double const out[4] = {agwn::div_rn_int(in[0], in[1]), agwn::sqrt_rn_int(in[0]), agwn::atan2_int(in[0], in[1]),
                               agwn::mul_rn_int(in[0], in[1])};
        std::fwrite(out, sizeof(double), 4, stdout);
    }
    return 0;
}
