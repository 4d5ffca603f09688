// Parametric fractional GWN over cubic Bezier boundary curves with adaptive G7-K15 quadrature:
// eval_gwnr_parametric_batch_fractional (src/antipodal/gwn_parametric.hh:168-186) with IntegratorGK15
// (src/antipodal/math/integrate_gk15.hh:63-290) and the integrand of gwn_parametric.hh:73-103.
//
// A panel is (depth, index): its end points are the dyadic numbers index * 2^-depth and its local tolerance
// tol * 2^-depth, exactly what the reference's halving computes, so a panel fits in 32 bits.  The tree is walked
// without recursion in the reference's order, and a finished left sibling's value per level replays its
// `left + right` summation (post-order).  Two arithmetic forms:
//  * exact -- the integrand and the G7/K15 sums in FP64, unfused, in the reference's order (k_param_exact): the
//    result equals the CPU reference bit for bit.
//  * mixed -- double-float arithmetic on the FP32 pipe (k_param_gk15).
//
// Proposal hook: a per-(query, curve) start depth s (from the learned proposal; 0 for the plain method).  Panels
// above depth s are split without being evaluated; every panel at depth >= s is evaluated and accepted or split by
// the reference's own rule.  When s does not exceed the shallowest leaf the plain method would accept, the two
// produce the same leaves and the same value; a larger s only refines further.

#include "agwn_internal.cuh"
#include "df32.cuh"
#include "hier.cuh"
#include "mlp.cuh"

#include <cmath>

namespace agwn
{
namespace
{
constexpr int kParamMaxDepth = 24; // deepest panel the integrator can reach (2^24 panels per curve)
constexpr int kParamBlock = 128;
// G7-K15 abscissae and weights: the published Gauss-Kronrod constants at the precision the reference carries
// (integrate_gk15.hh:13-36); identical doubles make the sums identical.
__constant__ double kGkX[8] = {0.0,
                               0.9914553711208126,
                               0.9491079123427585,
                               0.8648644233597691,
                               0.7415311855993945,
                               0.5860872354676911,
                               0.4058451513773972,
                               0.2077849550078985};
__constant__ double kGkWk[8] = {0.2094821410847278, 0.0229353220105292, 0.0630920926299786, 0.1047900103222502,
                                0.1406532597155259, 0.1690047266392679, 0.1903505780647854, 0.2044329400752989};
constexpr double kGkWgCenter = 0.4179591836734694;
constexpr double kGkWg2 = 0.1294849661688697;
constexpr double kGkWg4 = 0.2797053914892767;
constexpr double kGkWg6 = 0.3818300505051189;

struct dual
{
    rd v, d;
};
__device__ __forceinline__ dual dmul(dual a, dual b)
{
    return {a.v * b.v, a.d * b.v + a.v * b.d};
}
__device__ __forceinline__ dual smul(rd s, dual b)
{
    return {s * b.v, s * b.d};
}

// The cubic Bernstein polynomials and their derivatives at t, by the reference's dual-number evaluation: the values
// b0..b3, then the derivatives.
struct Bernstein
{
    rd v[4], d[4];
};
__device__ __forceinline__ Bernstein bernstein(double tt)
{
    dual const t{rd(tt), rd(1.0)};
    dual const u{rd(1.0) - rd(tt), rd(-1.0)};
    dual const b0 = dmul(dmul(u, u), u);
    dual const b1 = dmul(dmul(smul(rd(3.0), u), u), t);
    dual const b2 = dmul(dmul(smul(rd(3.0), u), t), t);
    dual const b3 = dmul(dmul(t, t), t);
    return {{b0.v, b1.v, b2.v, b3.v}, {b0.d, b1.d, b2.d, b3.d}};
}

// w(t) - d_eta(t) for the cubic Bezier curve c at the parameter of basis B (summed c0*b0 + c1*b1 + c2*b2 + c3*b3) and
// normalize_fd (src/antipodal/math/fwd_diff.hh:497-532).  The reference's x1 = -x0 appears negated: each of its
// products and sums is the exact negative of the one with x0, so b = -a, b' = -a', and x1 b = x0 a.
__device__ __forceinline__ double integrand(const double (&c)[12], Bernstein const& B, ev3<rd> p, ev3<rd> x0)
{
    rd phi[3], dphi[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
        phi[k] = rd(c[k]) * B.v[0] + rd(c[3 + k]) * B.v[1] + rd(c[6 + k]) * B.v[2] + rd(c[9 + k]) * B.v[3];
        dphi[k] = rd(c[k]) * B.d[0] + rd(c[3 + k]) * B.d[1] + rd(c[6 + k]) * B.d[2] + rd(c[9 + k]) * B.d[3];
    }
    ev3<rd> const r{phi[0] - p.x, phi[1] - p.y, phi[2] - p.z};
    ev3<rd> const dr{dphi[0], dphi[1], dphi[2]};
    rd const q = r.x * r.x + r.y * r.y + r.z * r.z;
    rd const q1 = rd(2.0) * (r.x * dr.x + r.y * dr.y + r.z * dr.z);
    rd const s = ex_sqrt(q);
    rd const inv_s = rd(1.0) / s;
    rd const s1 = q1 * (rd(0.5) * inv_s);
    ev3<rd> G, Gp;
    G.x = r.x * inv_s;
    G.y = r.y * inv_s;
    G.z = r.z * inv_s;
    Gp.x = (dr.x - G.x * s1) * inv_s;
    Gp.y = (dr.y - G.y * s1) * inv_s;
    Gp.z = (dr.z - G.z * s1) * inv_s;
    rd const a = edot(x0, G);
    rd const ap = edot(x0, Gp);
    // The products from here on take the integer pipe, beside the sums.  The two quotients have one form,
    // axis . (A x A') / |A|^2, and share their code (inlined twice, the products overflow the instruction cache).
    auto const i3 = [](ev3<rd> const& u) { return ev3<rdi>{rdi(u.x.v), rdi(u.y.v), rdi(u.z.v)}; };
    ev3<rdi> const g = i3(G), gp = i3(Gp), z = i3(x0);
    rdi const ai = rdi(a.v), api = rdi(ap.v);
    ev3<rdi> A = g - ev3<rdi>{z.x * ai, z.y * ai, z.z * ai};
    ev3<rdi> Ap = gp - ev3<rdi>{z.x * api, z.y * api, z.z * api};
    ev3<rdi> axis = z;
    ev3<rdi> const X = z - ev3<rdi>{g.x * ai, g.y * ai, g.z * ai};
    ev3<rdi> const Xp = ev3<rdi>{g.x * -api, g.y * -api, g.z * -api} - ev3<rdi>{gp.x * ai, gp.y * ai, gp.z * ai};
    rd w = rd(0.0), d_eta = rd(0.0);
#pragma unroll 1
    for (int term = 0; term < 2; ++term)
    {
        rd const quotient = rd((edot(axis, ecross(A, Ap)) / edot(A, A)).v);
        w = d_eta;
        d_eta = term == 0 ? -quotient : quotient; // first -x0 . (v x v') / |v|^2 = w, then G . (X x X') / |X|^2
        A = X;
        Ap = Xp;
        axis = g;
    }
    return (w - d_eta).v;
}

// ---- exact form -----------------------------------------------------------------------------------------------
// A panel's 15 nodes are the lanes of a team of 16 (half a warp): lane 0 the centre, lanes 1-7 the nodes
// centre - h x_k, lanes 8-14 centre + h x_(lane - 7), lane 15 a copy of the centre.
constexpr int kTeam = 16;
// The nodes' Bernstein bases depend on the panel alone, not on the curve or the query.  They are tabulated once per
// context down to this depth: double2 [panel 2^d - 1 + j][4][16 lanes], the four pairs (v0 v1), (v2 v3), (d0 d1),
// (d2 d3) -- 2.1 MB, read coalesced from L2, in place of 34 of the integrand's FP64 instructions.
constexpr int kBernDepth = 10;
constexpr int kBernPanels = (2 << kBernDepth) - 1;

__device__ __forceinline__ double node_x(int lane)
{
    return kGkX[lane == 15 ? 0 : (lane < 8 ? lane : lane - 7)];
}
__device__ __forceinline__ double pow2_neg(int e) // 2^-e
{
    return of_bits(uint64_t(1023 - e) << 52);
}
// The team's node of panel (depth, j) = [j 2^-depth, (j + 1) 2^-depth].
__device__ __forceinline__ double panel_node(int depth, uint32_t j, int lane, double xk)
{
    double const scale = pow2_neg(depth);
    double const aa = double(j) * scale, bb = double(j + 1) * scale; // exact: j < 2^24
    rd const cc = (rd(aa) + rd(bb)) * rd(0.5);
    rd const h = (rd(bb) - rd(aa)) * rd(0.5);
    rd const dx = h * rd(xk);
    return (lane < 8 ? cc - dx : cc + dx).v;
}

__global__ void k_bernstein(double2* __restrict__ table)
{
    int const i = int(blockIdx.x * blockDim.x + threadIdx.x), lane = i % kTeam, panel = i / kTeam;
    if (panel >= kBernPanels)
        return;
    int const d = 31 - __clz(panel + 1);
    Bernstein const B = bernstein(panel_node(d, uint32_t(panel + 1 - (1 << d)), lane, node_x(lane)));
    double2* const o = table + size_t(panel) * 4 * kTeam + lane;
    for (int k = 0; k < 2; ++k)
    {
        o[k * kTeam] = make_double2(B.v[2 * k].v, B.v[2 * k + 1].v);
        o[(k + 2) * kTeam] = make_double2(B.d[2 * k].v, B.d[2 * k + 1].v);
    }
}

// ---- double-float form ----------------------------------------------------------------------------------------
// The same integrand and panel rule in double-float arithmetic (df32.cuh, ~44 significant bits on the FP32 pipe):
// the curve relative to the query in power form about t = 1/2 (k_curves_df), in the frame of x0, and w - d_eta in
// the closed form below -- the same quantities in fewer operations.  Not bit-identical to the reference (the value differs in the
// last ~1e-13 relative, and a panel whose |Ik - Ig| sits at the tolerance can be decided the other way); the tree
// rule, the tolerances and the summation order are the plain integrator's.
struct alignas(16) CurveDF
{
    df c[12];
};

constexpr float hi_of(double d)
{
    return float(d);
}
constexpr float lo_of(double d)
{
    return float(d - double(float(d)));
}
#define AGWN_DF(d) {hi_of(d), lo_of(d)}
__constant__ df kGkXdf[8] = {AGWN_DF(0.0),
                             AGWN_DF(0.9914553711208126),
                             AGWN_DF(0.9491079123427585),
                             AGWN_DF(0.8648644233597691),
                             AGWN_DF(0.7415311855993945),
                             AGWN_DF(0.5860872354676911),
                             AGWN_DF(0.4058451513773972),
                             AGWN_DF(0.2077849550078985)};
__constant__ df kGkWkdf[8] = {AGWN_DF(0.2094821410847278), AGWN_DF(0.0229353220105292), AGWN_DF(0.0630920926299786),
                              AGWN_DF(0.1047900103222502), AGWN_DF(0.1406532597155259), AGWN_DF(0.1690047266392679),
                              AGWN_DF(0.1903505780647854), AGWN_DF(0.2044329400752989)};
__constant__ df kGkWgdf[4] = {AGWN_DF(0.4179591836734694), AGWN_DF(0.1294849661688697), AGWN_DF(0.2797053914892767),
                              AGWN_DF(0.3818300505051189)};
#undef AGWN_DF

__device__ __forceinline__ df df_mulf(df a, float f)
{
    df const p = two_prod(a.hi, f);
    return fast_two_sum(p.hi, __fmaf_rn(a.lo, f, p.lo));
}

// The frame of the double-float form: x0 along +z (rows e1, e2, x0 / |x0|).  Curves and queries are rotated into it in
// FP64 once per call, before their rounding to double-float.
struct FrameDF
{
    double r[9];
    df len;   // |x0|
    df scale; // (|x0|^2 - 2) |x0|^2
    bool unit;
};

// w(t) - d_eta(t) in closed form.  The exact kernel evaluates the reference's expression (integrand,
// gwn_parametric.hh:73-103): with G = r / |r|, G' its derivative, a = x0.G,
// X = x0 - G a, X' = -(G (x0.G') + G' a), v = G - x0 a, v' = G' - x0 (x0.G'), d_eta = G.(X x X') / |X|^2 and
// w = -x0.(v x v') / |v|^2.  Expanding (G x G = 0, G.(G x G') = 0, |G| = 1): G.(X x X') = a c and
// x0.(v x v') = c with c = x0.(G x G'), |X|^2 = n - a^2 = |x0 x G|^2 (Lagrange's identity) and
// |v|^2 = 1 + (n - 2) a^2 with n = |x0|^2.  In terms of r itself (s = |r|, q = s^2, m = x0.r, G x G' = r x r' / q,
// so c = T / q with T = x0.(r x r') = r'.(x0 x r)):
//   w - d_eta = -T / (q + (n - 2) m^2) - m T / (s |x0 x r|^2),
// and for a unit x0 (n = 1 to double precision) -T / (s (s - m)), free of the two terms' cancellation near
// m = -s.  Near m = s (the curve crossing the ray of x0 from the query) s - m, formed by subtraction, would keep
// only the square of the angle's relative precision; there it is |x0 x r|^2 / (s + m), whose squares keep the
// angle's own.  For a unit x0: one square root and one quotient, against the expression's square root and three
// quotients.
//
// In the frame with x0 = |x0| z these are two-term forms: m = |x0| z, T = |x0| (x y' - y x'), |x0 x r|^2 = n (x^2 + y^2),
// and z' is not needed.  A node takes about 370 FP32 operations; with x0's three coordinates it took about 660.  Errors
// against the exact form did not grow: p50 4.2e-15 -> 2.8e-15, p99 2.6e-11 -> 1.8e-11, p99.9 3.8e-10 -> 2.3e-10 over 4 x
// 30,000 queries, 30% of them within 1e-3 of a curve.  (Products that go into their sums without being normalised first
// would save 10% of the time, and lose half a bit of each.)
// pc: the pair's curve minus its query as power coefficients about t = 1/2 (k_curves_df), dl = t - 1/2.
__device__ __forceinline__ df integrand_df(const df (&pc)[12], FrameDF const& F, df dl)
{
    // r = a0 + dl (a1 + dl (a2 + dl a3)) by Horner's rule, and r' = a1 + dl (2 a2 + 3 dl a3) from its partial sums
    df r[3], d[2];
#pragma unroll
    for (int c = 0; c < 3; ++c)
    {
        df const t2 = df_fma(dl, pc[9 + c], pc[6 + c]);
        df const t1 = df_fma(dl, t2, pc[3 + c]);
        r[c] = df_fma(dl, t1, pc[c]);
        if (c < 2)
            d[c] = df_fma(dl, df_fma(dl, pc[9 + c], t2), t1);
    }
    df const rho = df_dot2(r[0], r[0], r[1], r[1]);
    df const q = df_fma(r[2], r[2], rho);
    df const s = df_sqrt(q);
    df const T = df_det2(r[0], d[1], r[1], d[0]);
    if (F.unit)
    {
        bool const behind = r[2].hi < 0.f;
        // s + |z|: s - m behind, s + m in front
        df const sm = df_add_ordered(s, behind ? df_neg(r[2]) : r[2]);
        df const num = T * sm;
        df const den = s * df{behind ? sm.hi : rho.hi, behind ? sm.lo : rho.lo};
        return df_neg(df{behind ? T.hi : num.hi, behind ? T.lo : num.lo} / den);
    }
    return df_neg(F.len * T / df_fma(F.scale, r[2] * r[2], q)) - (r[2] * T) / (s * rho);
}

__device__ __forceinline__ double gk15_panel_df(const df (&pc)[12], FrameDF const& F, int depth, uint32_t j, float* err)
{
    float const scale = ldexpf(1.f, -depth);
    float const h = 0.5f * scale;
    // the centre (j + 1/2) 2^-depth less 1/2: a multiple of 2^-(depth + 1) below 1/2 in magnitude, so a float exactly
    float const cc = __fadd_rn(__fmaf_rn(float(j), scale, -0.5f), h);
    df const f0 = integrand_df(pc, F, df_make(cc));
    // the Kronrod and Gauss sums accumulated node pair by node pair, in the order of the sums above (the same
    // values), so no node value stays live
    df ig = kGkWgdf[0] * f0;
    df ik = kGkWkdf[0] * f0;
#pragma unroll 1
    for (int k = 1; k <= 7; ++k)
    {
        df const dx = df_scale(kGkXdf[k], h);
        df const up = two_sum(cc, dx.hi), dn = two_sum(cc, -dx.hi);
        df const s = integrand_df(pc, F, fast_two_sum(dn.hi, __fsub_rn(dn.lo, dx.lo))) +
                     integrand_df(pc, F, fast_two_sum(up.hi, __fadd_rn(up.lo, dx.lo)));
        ik = df_fma(kGkWkdf[k], s, ik);
        if ((k & 1) == 0)
            ig = df_fma(kGkWgdf[k >> 1], s, ig);
    }
    df const diff = df_scale(ik - ig, h);
    *err = fabsf(diff.hi + diff.lo);
    return df_to(df_scale(ik, h));
}

// Queries in the frame, as double-float coordinates.
__global__ void k_queries_df(const double* __restrict__ pts, int64_t n, FrameDF F, df* __restrict__ out)
{
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    {
        double const x = pts[3 * i], y = pts[3 * i + 1], z = pts[3 * i + 2];
        for (int c = 0; c < 3; ++c)
            out[3 * i + c] = df_from(F.r[3 * c] * x + F.r[3 * c + 1] * y + F.r[3 * c + 2] * z);
    }
}

// Curves in the frame, as power coefficients about t = 1/2: with s03 = c0 + c3, s12 = c1 + c2, d30 = c3 - c0 and
// d21 = c2 - c1, r(1/2) = (s03 + 3 s12) / 8, r'(1/2) = 3/4 (d30 + d21), r^(2)(1/2) / 2 = 3/2 (s03 - s12) and
// r^(3) / 6 = d30 - 3 d21, formed in FP64 and rounded to double-float once.  A query enters r(1/2) only, so a pair
// subtracts three coordinates.  (Evaluated at |t - 1/2| <= 1/2 the power form rounds a little worse than the Bernstein
// form: in FP32 on bicubic patch boundaries, relative error of r, median 1.2x at random pairs with a lower maximum,
// median 1.7x and p99 2.1x for queries 1e-4 to 1e-2 from a curve near their closest point.)
__global__ void k_curves_df(const double* __restrict__ curves, int64_t n_curves, FrameDF F, CurveDF* __restrict__ out)
{
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < 3 * n_curves;
         i += int64_t(gridDim.x) * blockDim.x)
    {
        int64_t const k = i / 3;
        int const c = int(i - 3 * k);
        const double* const v = curves + 12 * k;
        double p[4];
        for (int e = 0; e < 4; ++e)
            p[e] = F.r[3 * c] * v[3 * e] + F.r[3 * c + 1] * v[3 * e + 1] + F.r[3 * c + 2] * v[3 * e + 2];
        double const s03 = p[0] + p[3], s12 = p[1] + p[2], d30 = p[3] - p[0], d21 = p[2] - p[1];
        df* const o = out[k].c + c;
        o[0] = df_from(0.125 * (s03 + 3.0 * s12));
        o[3] = df_from(0.75 * (d30 + d21));
        o[6] = df_from(1.5 * (s03 - s12));
        o[9] = df_from(d30 - 3.0 * d21);
    }
}

// Optional work of the integrator kernel.
//   panel_log: training data for the per-panel network, 2 words per evaluated panel below max_depth -- the pair's
//     index (query * n_curves + curve) and (depth << 25) | (j << 1) | accepted; entries past log_cap are counted,
//     not written.
//   pwb / pparams (double-float kernel only): the per-panel network.  Before a panel below max_depth is evaluated
//     the warp runs the network on its lanes' panels; a panel whose predicted chance of being accepted is below
//     beta (logit margin < skip_logit) is split without evaluation.  Every evaluated panel is still accepted or split
//     by the plain error test.
struct ParamExtras
{
    uint32_t* panel_log;
    unsigned long long* log_count;
    long long log_cap;
    const __nv_bfloat16* pwb;
    const float* pparams;
    float skip_logit;
    float log10_tol;
    unsigned long long* skip_count;
};

// Pair integrals in the exact form: vals[k * nq + i] for the curves c0 + k and the queries q0 + i.
//
// FP64 issue bounds it (one warp instruction per 16 clocks per SM; about 155 for an integrand of 15 nodes x 2 panels,
// and 12 for a panel's sums).  The cost of one pair is heavy-tailed -- a query whose line along x0 passes close to a
// curve needs a deep tree there -- so the teams of the whole grid draw their pairs from one counter, and a panel takes
// one integrand time, not 15: a deep pair is no tail, and a few pairs fill the chip.  Each team walks its pair's panel
// tree without a stack: after a split the next panel is the left child (depth + 1, 2j); after an accepted leaf the
// walk climbs while the finished node is a right child (j odd), combining left + right from `pending` (the finished
// left sibling's value per level), then moves to the right sibling (depth, j + 1).  Panels above the pair's start
// depth are not evaluated: the walk descends to the leftmost descendant at the start depth.  All lanes of a team hold
// the same walk state.  Measured against one thread per pair with the pairs of 128 queries on one block: 3,001
// queries x 96 curves at tol 1e-8 (24 such blocks) 86.5 -> 9.5 ms.
__global__ void __launch_bounds__(kParamBlock, 4)
    k_param_exact(const double* __restrict__ pos, int64_t q0, int nq, ev3<rd> x0, const double* __restrict__ curves,
                  int64_t n_curves, int64_t c0, int nc, int min_depth, int max_depth, double tol,
                  const uint8_t* __restrict__ start_depth, uint32_t* __restrict__ stats, int32_t* __restrict__ nodes_total,
                  double* __restrict__ vals, int* __restrict__ next, const double2* __restrict__ table, ParamExtras ex)
{
    __shared__ double tol_at[kParamMaxDepth + 1];
    __shared__ double s_pending[kParamBlock / kTeam][kParamMaxDepth + 1];
    if (threadIdx.x == 0)
    {
        // tol * 2^-d by repeated halving, as the recursion computes it (exact unless it reaches subnormals)
        tol_at[0] = tol;
        for (int l = 1; l <= kParamMaxDepth; ++l)
            tol_at[l] = __dmul_rn(tol_at[l - 1], 0.5);
    }
    __syncthreads();
    int const total = nq * nc;
    unsigned const lane = threadIdx.x & 31u, tm = 0xffffu << (lane & 16u);
    int const tl = int(lane & 15u);
    double const xk = node_x(tl);
    // lanes 0-7 weigh the node sums for Ik, lanes 8-15 (the same sums again) for Ig: 0 at the odd ones
    double const wt = tl < 8 ? kGkWk[tl]
                             : (tl == 8 ? kGkWgCenter : tl == 10 ? kGkWg2 : tl == 12 ? kGkWg4 : tl == 14 ? kGkWg6 : 0.0);
    bool const weighed = tl < 8 || (tl & 1) == 0;
    double* const pending = s_pending[threadIdx.x / kTeam];
    int pi = -1; // this team's pair, -1 = needs one
    bool drained = false;
    int k = 0, ql = 0, s = 0, d = 0, leaves = 0, dmin = 0, dmax = 0, pnodes = 0;
    uint32_t j = 0;
    ev3<rd> p{};
    double c[12] = {};
    for (;;)
    {
        unsigned const want = __ballot_sync(0xffffffffu, tl == 0 && pi < 0 && !drained);
        if (want)
        {
            int base = 0;
            if (lane == 0)
                base = atomicAdd(next, __popc(want));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (pi < 0 && !drained)
            {
                int const mine = base + __popc(want & ((1u << (lane & 16u)) - 1u));
                if (mine < total)
                {
                    pi = mine;
                    k = mine / nq;
                    ql = mine - k * nq;
                    int64_t const q = q0 + ql;
                    p = ev3<rd>{rd(pos[3 * q]), rd(pos[3 * q + 1]), rd(pos[3 * q + 2])};
                    const double* const cv = curves + 12 * (c0 + k);
#pragma unroll
                    for (int e = 0; e < 12; ++e)
                        c[e] = cv[e];
                    s = start_depth ? min(int(start_depth[q * n_curves + c0 + k]), max_depth) : 0;
                    d = s;
                    j = 0;
                    leaves = 0;
                    dmin = 255;
                    dmax = 0;
                    pnodes = 0;
                }
                else
                    drained = true;
            }
        }
        if (!__any_sync(0xffffffffu, pi >= 0))
            break;
        if (pi >= 0) // the team's lanes agree
        {
            rd const h = rd(pow2_neg(d + 1)); // half the panel's width, exact
            Bernstein B;
            if (d <= kBernDepth)
            {
                const double2* const r = table + size_t((1u << d) - 1u + j) * 4 * kTeam + tl;
                double2 const b0 = __ldg(r), b1 = __ldg(r + kTeam), b2 = __ldg(r + 2 * kTeam), b3 = __ldg(r + 3 * kTeam);
                B = {{rd(b0.x), rd(b0.y), rd(b1.x), rd(b1.y)}, {rd(b2.x), rd(b2.y), rd(b3.x), rd(b3.y)}};
            }
            else
                B = bernstein(panel_node(d, j, tl, xk));
            double const f = integrand(c, B, p, x0);
            // the sums of the reference (integrate_gk15.hh:155-217): s_0 = f(centre), s_k = f(-k) + f(+k), then
            // Ik = (wk_0 s_0 + wk_1 s_1 + ...) h term by term, Ig likewise over the even k (lanes 8-15 add exact
            // zeros for the others)
            double const other = __shfl_sync(tm, f, (tl & 7) + 7, kTeam);
            double const mine = __shfl_sync(tm, f, tl & 7, kTeam);
            double const sum2 = (tl & 7) ? (rd(mine) + rd(other)).v : mine;
            double const term = weighed ? (rd(wt) * rd(sum2)).v : 0.0;
            rd acc = rd(__shfl_sync(tm, term, tl & 8, kTeam));
#pragma unroll
            for (int e = 1; e < 8; ++e)
                acc = acc + rd(__shfl_sync(tm, term, (tl & 8) + e, kTeam));
            acc = acc * h;
            double const twin = __shfl_xor_sync(tm, acc.v, 8, kTeam);
            double const err = fabs((acc - rd(twin)).v);
            double v = tl < 8 ? acc.v : twin;
            ++pnodes;
            bool const accept = d >= max_depth || (d >= min_depth && err <= tol_at[d]);
            if (ex.panel_log && d < max_depth && tl == 0)
            {
                unsigned long long const slot = atomicAdd(ex.log_count, 1ull);
                if ((long long)slot < ex.log_cap)
                {
                    ex.panel_log[2 * slot] = uint32_t((q0 + ql) * n_curves + c0 + k);
                    ex.panel_log[2 * slot + 1] = (uint32_t(d) << 25) | (j << 1) | (accept ? 1u : 0u);
                }
            }
            if (!accept)
            {
                ++d; // split: left child next
                j <<= 1;
            }
            else
            {
                ++leaves;
                dmin = min(dmin, d);
                dmax = max(dmax, d);
                while (d > 0 && (j & 1u))
                {
                    v = __dadd_rn(pending[d], v); // left + right
                    --d;
                    j >>= 1;
                }
                if (d > 0)
                {
                    pending[d] = v; // a finished left child (every lane stores the same value): its sibling is next
                    ++j;
                    while (d < s)
                    {
                        ++d;
                        j <<= 1;
                    }
                }
                else
                {
                    // the root is done: v is this pair's integral
                    if (tl == 0)
                    {
                        vals[int64_t(k) * nq + ql] = v;
                        if (stats)
                            stats[(q0 + ql) * n_curves + c0 + k] = uint32_t(min(leaves, 0xffff)) |
                                                                   (uint32_t(dmin) << 16) | (uint32_t(dmax) << 24);
                        if (nodes_total)
                            atomicAdd(nodes_total + q0 + ql, pnodes);
                    }
                    pi = -1;
                }
            }
        }
        __syncwarp();
    }
}

// The pair integrals of each query added in curve order: out[i] (the running sum, from 0 with `first`) over this
// chunk's curves, divided by 4 pi with `last`.
__global__ void k_param_sum(const double* __restrict__ vals, int nq, int nc, bool first, bool last,
                            double* __restrict__ out)
{
    int const i = int(blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= nq)
        return;
    rd sum = first ? rd(0.0) : rd(out[i]);
#pragma unroll 8
    for (int k = 0; k < nc; ++k)
        sum = sum + rd(vals[int64_t(k) * nq + i]);
    out[i] = last ? (sum / (rd(4.0) * rd(3.141592653589793238462643383279502884))).v : sum.v;
}

// Pair integrals in the double-float form: vals[k * nq + i] for the curves c0 + k and the queries q0 + i (pos: these
// queries' coordinates).
//
// The FMA pipe's chains bound it (a lane per pair: some 370 dependent FP32 operations a node, 15 nodes a panel).  The
// cost of one (query, curve) integral is heavy-tailed, so the lanes of the whole grid draw their pairs from one counter
// (a warp takes `take`, 32 or 64, at a time) and walk their panel trees as a team of the exact form does; k_param_sum adds a
// query's integrals in curve order.  With blocks of 128 queries x 128 curves as the unit, 20,000 queries x 1,024 curves
// made 1.4 waves of them and each block waited for its deepest pair: the whole call 34.5 -> 31.5 ms.
//
// start_depth: per (query, curve), row-major [n][n_curves], nullable = all 0.  stats (nullable): per (query,
// curve) packed as leaves | shallowest leaf depth << 16 | deepest leaf depth << 24.  nodes_total (nullable, zeroed):
// panels evaluated per query.
// The per-panel network's shared memory.
struct PanelSmem
{
    WeightsSmem w;
    uint32_t feat[kParamBlock / 32][32][kS16 - 4 + 1];
    float logit[kParamBlock / 32][32][2];
};

// PANEL: the per-panel network runs (its code and shared memory are compiled only into this instance, so the other
// instance keeps its registers).
template <bool PANEL>
constexpr int param_min_blocks()
{
    return !PANEL ? 6 : 1; // the double-float panels in 80 registers (no spills), six blocks per SM
}
template <bool PANEL>
__global__ void __launch_bounds__(kParamBlock, param_min_blocks<PANEL>())
    k_param_gk15(const df* __restrict__ pos, int64_t q0, int nq, FrameDF F, const CurveDF* __restrict__ curves,
                 int64_t n_curves, int64_t c0, int nc, int min_depth, int max_depth, double tol,
                 const uint8_t* __restrict__ start_depth, uint32_t* __restrict__ stats,
                 int32_t* __restrict__ nodes_total, double* __restrict__ vals, int* __restrict__ next, int take,
                 ParamExtras ex)
{
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ double tol_at[kParamMaxDepth + 1];
    PanelSmem* const ps = reinterpret_cast<PanelSmem*>(smem);
    bool const use_panel = PANEL && ex.pwb != nullptr;
    unsigned long long skips = 0;
    unsigned const lane = threadIdx.x & 31u;
    if (threadIdx.x == 0)
    {
        // tol * 2^-depth by repeated halving, as the recursion computes it (exact unless it reaches subnormals)
        tol_at[0] = tol;
        for (int l = 1; l <= kParamMaxDepth; ++l)
            tol_at[l] = __dmul_rn(tol_at[l - 1], 0.5);
    }
    if (use_panel)
        load_weights(ps->w, ex.pwb, ex.pparams);
    float3 const x0f = make_float3(0.f, 0.f, F.len.hi);
    int const warp = int(threadIdx.x >> 5);
    __syncthreads();
    int const total = nc * nq; // curve-major
    int taken = 0, end = 0;    // this warp's pairs not yet given to a lane: [taken, end)
    int pi = -1;                // this lane's pair, -1 = needs one
    bool drained = false;
    int k = 0, ql = 0, s = 0, d = 0, leaves = 0, dmin = 0, dmax = 0, pnodes = 0;
    uint32_t j = 0;
    df cp[12]; // this pair's curve minus its query, as power coefficients about t = 1/2
    double pending[kParamMaxDepth + 1];
    for (;;)
    {
        unsigned const want = __ballot_sync(0xffffffffu, pi < 0 && !drained);
        if (want)
        {
            int const need = __popc(want), left = end - taken, rank = __popc(want & ((1u << lane) - 1u));
            int fresh = 0;
            if (left < need)
            {
                if (lane == 0)
                    fresh = atomicAdd(next, take);
                fresh = __shfl_sync(0xffffffffu, fresh, 0);
            }
            if (want & (1u << lane))
            {
                int const mine = rank < left ? taken + rank : fresh + rank - left;
                if (mine < total)
                {
                    pi = mine;
                    k = mine / nq;
                    ql = mine - k * nq;
                    int64_t const q = q0 + ql;
                    df const pd[3] = {pos[3 * ql], pos[3 * ql + 1], pos[3 * ql + 2]};
                    CurveDF const& cv = curves[c0 + k];
#pragma unroll
                    for (int e = 0; e < 12; ++e)
                        cp[e] = e < 3 ? cv.c[e] - pd[e] : cv.c[e];
                    s = start_depth ? min(int(start_depth[q * n_curves + c0 + k]), max_depth) : 0;
                    d = s;
                    j = 0;
                    leaves = 0;
                    dmin = 255;
                    dmax = 0;
                    pnodes = 0;
                }
                else
                    drained = true;
            }
            taken = left < need ? fresh + need - left : taken + need;
            end = left < need ? fresh + take : end;
        }
        if (!__any_sync(0xffffffffu, pi >= 0))
            break;
        // the per-panel network: up to four rounds of "split it without evaluating", all lanes together
        for (int round = 0; PANEL && use_panel && round < 4; ++round)
        {
            bool const cand = pi >= 0 && d < max_depth;
            float f[kF];
            if (cand)
            {
                // the control points minus the query, as the network was trained on them: a0 -+ a1/2 + a2/4
                // -+ a3/8 at the ends, a0 -+ a1/6 - a2/12 +- a3/8 between
                float cpf[12];
#pragma unroll
                for (int e = 0; e < 3; ++e)
                {
                    df const o1 = df_mulf(cp[3 + e], 1.f / 6.f), e2 = df_mulf(cp[6 + e], 1.f / 12.f);
                    df const end = cp[e] + df_scale(cp[6 + e], 0.25f), mid = cp[e] - e2;
                    df const a3 = df_scale(cp[9 + e], 0.125f), odd = df_scale(cp[3 + e], 0.5f) + a3;
                    cpf[e] = (end - odd).hi;
                    cpf[3 + e] = (mid - o1 + a3).hi;
                    cpf[6 + e] = (mid + o1 - a3).hi;
                    cpf[9 + e] = (end + odd).hi;
                }
                panel_features(cpf, d, j, x0f, ex.log10_tol, f);
            }
            else
            {
#pragma unroll
                for (int e = 0; e < kF; ++e)
                    f[e] = 0.f;
            }
            uint32_t* const row = ps->feat[warp][lane];
#pragma unroll
            for (int e = 0; e < kF / 2; ++e)
                row[e] = pack_bf16(f[2 * e], f[2 * e + 1]);
            row[6] = 0u;
            row[7] = 0u;
            __syncwarp();
            int const g = int(lane >> 2), tig = int(lane & 3u);
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
            {
                uint32_t a0[4] = {ps->feat[warp][mt * 16 + g][tig], ps->feat[warp][mt * 16 + g + 8][tig],
                                  ps->feat[warp][mt * 16 + g][4 + tig],
                                  ps->feat[warp][mt * 16 + g + 8][4 + tig]};
                float z1[8][4], z2[8][4], z3[2][4];
                mlp_forward(ps->w, a0, z1, z2, z3);
                if (tig == 0) // columns 0 and 1: the split and accept logits
                {
                    ps->logit[warp][mt * 16 + g][0] = z3[0][0];
                    ps->logit[warp][mt * 16 + g][1] = z3[0][1];
                    ps->logit[warp][mt * 16 + g + 8][0] = z3[0][2];
                    ps->logit[warp][mt * 16 + g + 8][1] = z3[0][3];
                }
            }
            __syncwarp();
            bool const skip =
                cand && (ps->logit[warp][lane][1] - ps->logit[warp][lane][0]) < ex.skip_logit;
            __syncwarp();
            if (!__any_sync(0xffffffffu, skip))
                break;
            if (skip)
            {
                ++d; // split without evaluating: left child next
                j <<= 1;
                ++skips;
            }
        }
        if (pi < 0)
            continue;
        float e32;
        double v = gk15_panel_df(cp, F, d, j, &e32);
        double const err = double(e32);
        ++pnodes;
        bool const accept = d >= max_depth || (d >= min_depth && err <= tol_at[d]);
        if (ex.panel_log && d < max_depth)
        {
            unsigned long long const slot = atomicAdd(ex.log_count, 1ull);
            if ((long long)slot < ex.log_cap)
            {
                ex.panel_log[2 * slot] = uint32_t((q0 + ql) * n_curves + c0 + k);
                ex.panel_log[2 * slot + 1] = (uint32_t(d) << 25) | (j << 1) | (accept ? 1u : 0u);
            }
        }
        if (!accept)
        {
            ++d; // split: left child next
            j <<= 1;
            continue;
        }
        ++leaves;
        dmin = min(dmin, d);
        dmax = max(dmax, d);
        while (d > 0 && (j & 1u))
        {
            v = __dadd_rn(pending[d], v); // left + right
            --d;
            j >>= 1;
        }
        if (d > 0)
        {
            pending[d] = v; // a finished left child: its right sibling is next
            ++j;
            while (d < s)
            {
                ++d;
                j <<= 1;
            }
            continue;
        }
        // the root is done: v is this pair's integral
        vals[int64_t(k) * nq + ql] = v;
        if (stats)
            stats[(q0 + ql) * n_curves + c0 + k] = uint32_t(min(leaves, 0xffff)) | (uint32_t(dmin) << 16) |
                                                   (uint32_t(dmax) << 24);
        if (nodes_total)
            atomicAdd(nodes_total + q0 + ql, pnodes);
        pi = -1;
    }
    if (ex.skip_count && skips)
        atomicAdd(ex.skip_count, skips);
}

// The pair integrals and their sums over chunks of at most `most` pairs: queries first, and curves where one query has
// more.  launch(q0, nq, c0, nc, vals, next) integrates a chunk's pairs.  reserve(nq) takes what else a chunk of nq queries
// needs.  Where there is no memory for a chunk, it is halved until there is.
template <class Reserve, class Launch>
int param_chunks(Context& ctx, int64_t n, int64_t n_curves, int64_t most, double* d_out, int32_t* d_nodes,
                 Reserve reserve, Launch launch)
{
    int64_t nc_max = 0, nq_max = 0;
    double* vals = nullptr;
    int* next = nullptr;
    AGWN_TRY(ctx.scratch_reserve(S_PARTIAL, sizeof(int), reinterpret_cast<void**>(&next)));
    most = std::min<int64_t>(most, n > most / n_curves ? most : n * n_curves);
    for (;; most /= 2)
    {
        nc_max = std::min(n_curves, most);
        nq_max = std::min(n, std::max<int64_t>(1, most / nc_max));
        int s = ctx.scratch_reserve(S_SEGS_RAW, sizeof(double) * size_t(nc_max) * size_t(nq_max),
                                    reinterpret_cast<void**>(&vals));
        if (s == AGWN_OK)
            s = reserve(nq_max);
        if (s == AGWN_OK)
            break;
        if (s != AGWN_ERR_NOMEM || most == 1)
            return s;
        // the larger buffers of this attempt or an earlier call make room
        clear_message();
        AGWN_TRY_CUDA(cudaStreamSynchronize(ctx.stream));
        ctx.scratch_drop(S_SEGS_RAW);
        ctx.scratch_drop(S_FRAME);
    }
    if (d_nodes)
        AGWN_TRY_CUDA(cudaMemsetAsync(d_nodes, 0, sizeof(int32_t) * n, ctx.stream));
    for (int64_t q0 = 0; q0 < n; q0 += nq_max)
        for (int64_t c0 = 0; c0 < n_curves; c0 += nc_max)
        {
            int const nq = int(std::min(nq_max, n - q0)), nc = int(std::min(nc_max, n_curves - c0));
            AGWN_TRY_CUDA(cudaMemsetAsync(next, 0, sizeof(int), ctx.stream));
            AGWN_TRY(launch(q0, nq, c0, nc, vals, next));
            AGWN_TRY(ctx.launch_begin(AGWN_K_OTHER));
            k_param_sum<<<div_up(nq, 64), 64, 0, ctx.stream>>>(vals, nq, nc, c0 == 0, c0 + nc == n_curves, d_out + q0);
            AGWN_TRY(ctx.launch_end(AGWN_K_OTHER));
        }
    return AGWN_OK;
}

// The exact form, 2^25 pairs (268 MB of integrals) at a time.
int param_run_exact(Context& ctx, const double* d_pos, int64_t n, double* d_out, const double* x0, const double* d_curves,
                    int64_t n_curves, int min_depth, int max_depth, double tol, const uint8_t* d_start,
                    uint32_t* d_stats, int32_t* d_nodes, ParamExtras const& ex)
{
    if (!ctx.bernstein_filled)
    {
        AGWN_TRY(ctx.bernstein.reserve(sizeof(double2) * 4 * kTeam * kBernPanels));
        AGWN_TRY(ctx.launch_begin(AGWN_K_OTHER));
        k_bernstein<<<div_up(kBernPanels * kTeam, 256), 256, 0, ctx.stream>>>(static_cast<double2*>(ctx.bernstein.ptr));
        AGWN_TRY(ctx.launch_end(AGWN_K_OTHER));
        // a launch that is being captured fills the table when the graph runs, not now
        cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
        AGWN_TRY_CUDA(cudaStreamIsCapturing(ctx.stream, &status));
        ctx.bernstein_filled = status == cudaStreamCaptureStatusNone;
    }
    int per_sm = 0;
    AGWN_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_param_exact, kParamBlock, 0));
    int64_t const full = int64_t(std::max(per_sm, 1)) * ctx.sm_count;
    ev3<rd> const x0v{rd(x0[0]), rd(x0[1]), rd(x0[2])};
    return param_chunks(
        ctx, n, n_curves, int64_t(1) << 25, d_out, d_nodes, [](int64_t) { return int(AGWN_OK); },
        [&](int64_t q0, int nq, int64_t c0, int nc, double* vals, int* next) -> int
        {
            int const grid = int(std::min<int64_t>(div_up(int64_t(nq) * nc, kParamBlock / kTeam), full));
            AGWN_TRY(ctx.launch_begin(AGWN_K_PARAMETRIC));
            k_param_exact<<<grid, kParamBlock, 0, ctx.stream>>>(d_pos, q0, nq, x0v, d_curves, n_curves, c0, nc, min_depth,
                                                               max_depth, tol, d_start, d_stats, d_nodes, vals, next,
                                                               static_cast<const double2*>(ctx.bernstein.ptr), ex);
            return ctx.launch_end(AGWN_K_PARAMETRIC);
        });
}
} // namespace

int param_run(Context& ctx, const double* d_pos, int64_t n, double* d_out, const double* x0, const double* d_curves,
              int64_t n_curves, int min_depth, int max_depth, double tol, const uint8_t* d_start, uint32_t* d_stats,
              int32_t* d_nodes, uint32_t* d_panel_log, unsigned long long* d_log_count, long long log_cap)
{
    bool const dfm = ctx.param_mode == AGWN_PARAM_MIXED;
    bool const panel = dfm && ctx.panel_mlp && tol > 0;
    ParamExtras ex{};
    ex.panel_log = d_panel_log;
    ex.log_count = d_log_count;
    ex.log_cap = log_cap;
    if (panel)
    {
        const void* wb = nullptr;
        mlp_device_weights(ctx.panel_mlp, &wb, &ex.pparams);
        ex.pwb = static_cast<const __nv_bfloat16*>(wb);
        double const b = std::min(std::max(double(ctx.panel_beta), 1e-9), 1.0 - 1e-9);
        ex.skip_logit = float(std::log(b / (1.0 - b)));
        ex.log10_tol = float(std::log10(tol));
        ex.skip_count = ctx.timing ? reinterpret_cast<unsigned long long*>(ctx.d_counters + 2) : nullptr;
    }
    if (n == 0)
        return AGWN_OK;
    if (n_curves == 0)
    {
        AGWN_TRY_CUDA(cudaMemsetAsync(d_out, 0, sizeof(double) * n, ctx.stream));
        if (d_nodes)
            AGWN_TRY_CUDA(cudaMemsetAsync(d_nodes, 0, sizeof(int32_t) * n, ctx.stream));
        return AGWN_OK;
    }
    if (!dfm)
        return param_run_exact(ctx, d_pos, n, d_out, x0, d_curves, n_curves, min_depth, max_depth, tol, d_start,
                               d_stats, d_nodes, ex);
    auto const kern = panel ? k_param_gk15<true> : k_param_gk15<false>;
    size_t const smem = panel ? sizeof(PanelSmem) : 0;
    AGWN_TRY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    int per_sm = 0;
    AGWN_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kParamBlock, smem));
    if (per_sm < 1)
        return fail(AGWN_ERR_UNSUPPORTED, "parametric kernel does not fit on an SM");
    int64_t const full = int64_t(per_sm) * ctx.sm_count;
    // curves and queries in the frame of x0, as double-floats
    FrameDF F;
    {
        Frame64 const f = ray_frame(x0);
        double const n2 = x0[0] * x0[0] + x0[1] * x0[1] + x0[2] * x0[2], len = std::sqrt(n2);
        auto const split = [](double v) { return df{float(v), float(v - double(float(v)))}; };
        for (int k = 0; k < 9; ++k)
            F.r[k] = f.r[k];
        F.len = split(len);
        F.scale = split((n2 - 2.0) * n2);
        F.unit = std::fabs(n2 - 1.0) <= 1e-15;
    }
    // the curves, then a chunk's queries
    CurveDF* cdf = nullptr;
    auto const reserve = [&](int64_t nq)
    {
        return ctx.scratch_reserve(S_FRAME, sizeof(CurveDF) * size_t(n_curves) + sizeof(df) * 3 * size_t(nq),
                                   reinterpret_cast<void**>(&cdf));
    };
    bool curves_done = false;
    // 2^26 pairs (537 MB of integrals) at a time: a chunk ends with its deepest pairs, half a millisecond or so
    return param_chunks(
        ctx, n, n_curves, int64_t(1) << 26, d_out, d_nodes, reserve,
        [&](int64_t q0, int nq, int64_t c0, int nc, double* vals, int* next) -> int
        {
            df* const qdf = reinterpret_cast<df*>(cdf + n_curves);
            if (!curves_done)
            {
                AGWN_TRY(ctx.launch_begin(AGWN_K_OTHER));
                k_curves_df<<<int(std::min<int64_t>(div_up(3 * n_curves, 256), 4 * ctx.sm_count)), 256, 0, ctx.stream>>>(
                    d_curves, n_curves, F, cdf);
                AGWN_TRY(ctx.launch_end(AGWN_K_OTHER));
                curves_done = true;
            }
            if (c0 == 0)
            {
                AGWN_TRY(ctx.launch_begin(AGWN_K_OTHER));
                k_queries_df<<<int(std::min<int64_t>(div_up(nq, 256), 4 * ctx.sm_count)), 256, 0, ctx.stream>>>(
                    d_pos + 3 * q0, nq, F, qdf);
                AGWN_TRY(ctx.launch_end(AGWN_K_OTHER));
            }
            int64_t const pairs = int64_t(nq) * nc;
            int const grid = int(std::min<int64_t>(div_up(pairs, kParamBlock), full));
            int const take = pairs >= 8 * full * kParamBlock ? 64 : 32;
            AGWN_TRY(ctx.launch_begin(AGWN_K_PARAMETRIC));
            kern<<<grid, kParamBlock, smem, ctx.stream>>>(qdf, q0, nq, F, cdf, n_curves, c0, nc, min_depth, max_depth, tol,
                                                         d_start, d_stats, d_nodes, vals, next, take, ex);
            return ctx.launch_end(AGWN_K_PARAMETRIC);
        });
}
} // namespace agwn

using namespace agwn;

namespace
{
// The parametric entry points: stage, optionally propose start depths with the learned network (mlp != NULL), run
// the integrator, copy host outputs back.
int param_entry(agwn_context* ctx, const agwn_mlp* mlp, int n_classes, float alpha, const double* positions, int64_t n,
                double* out, const double* x0, const double* curves, int64_t n_curves, int min_depth, int max_depth,
                double tol, const uint8_t* start_depth, uint32_t* pair_stats, int32_t* nodes_per_query)
{
    AGWN_CHECK_ARG(ctx && x0, "null context/x0");
    AGWN_CHECK_ARG(n >= 0 && n_curves >= 0 && (n == 0 || (positions && out)) && (n_curves == 0 || curves),
                   "bad arguments");
    AGWN_CHECK_ARG(min_depth >= 0 && max_depth >= 0 && max_depth <= kParamMaxDepth,
                   "depths must be in [0, %d] (max_depth bounds the explicit stack)", kParamMaxDepth);
    AGWN_CHECK_ARG(std::isfinite(tol) && tol >= 0, "tol must be finite and >= 0");
    AGWN_CHECK_ARG(n_curves < (int64_t(1) << 31), "too many curves");
    AGWN_CHECK_ARG(!mlp || tol > 0, "the learned proposal needs tol > 0");
    clear_message();
    AGWN_TRY_CUDA(cudaSetDevice(ctx->device));
    if (n == 0)
        return AGWN_OK;
    const void *dpos = nullptr, *dcur = nullptr, *dstart = nullptr;
    void *dout = nullptr, *dstats = nullptr, *dnodes = nullptr;
    bool h_out = false, h_stats = false, h_nodes = false;
    AGWN_TRY(stage_in(*ctx, positions, sizeof(double) * 3 * n, S_QUERIES, &dpos));
    AGWN_TRY(stage_in(*ctx, curves, sizeof(double) * 12 * n_curves, S_MISC0, &dcur));
    if (start_depth)
        AGWN_TRY(stage_in(*ctx, start_depth, size_t(n) * n_curves, S_MISC1, &dstart));
    AGWN_TRY(stage_out(*ctx, out, sizeof(double) * n, S_OUT, &dout, &h_out));
    if (pair_stats)
        AGWN_TRY(stage_out(*ctx, pair_stats, sizeof(uint32_t) * size_t(n) * n_curves, S_MISC2, &dstats, &h_stats));
    if (nodes_per_query)
        AGWN_TRY(stage_out(*ctx, nodes_per_query, sizeof(int32_t) * n, S_COUNTS, &dnodes, &h_nodes));
    if (mlp && n_curves > 0)
    {
        void* proposed = nullptr;
        AGWN_TRY(ctx->scratch_reserve(S_MISC1, size_t(n) * n_curves, &proposed));
        AGWN_TRY(mlp_propose_run(*ctx, mlp, static_cast<const double*>(dpos), n, x0, static_cast<const double*>(dcur),
                                 n_curves, n_classes, min_depth, max_depth, tol, alpha,
                                 static_cast<uint8_t*>(proposed), nullptr));
        dstart = proposed;
    }
    AGWN_TRY(param_run(*ctx, static_cast<const double*>(dpos), n, static_cast<double*>(dout), x0,
                       static_cast<const double*>(dcur), n_curves, min_depth, max_depth, tol,
                       static_cast<const uint8_t*>(dstart), static_cast<uint32_t*>(dstats),
                       static_cast<int32_t*>(dnodes)));
    if (h_out)
        AGWN_TRY_CUDA(cudaMemcpyAsync(out, dout, sizeof(double) * n, cudaMemcpyDeviceToHost, ctx->stream));
    if (h_stats)
        AGWN_TRY_CUDA(cudaMemcpyAsync(pair_stats, dstats, sizeof(uint32_t) * size_t(n) * n_curves,
                                      cudaMemcpyDeviceToHost, ctx->stream));
    if (h_nodes)
        AGWN_TRY_CUDA(cudaMemcpyAsync(nodes_per_query, dnodes, sizeof(int32_t) * n, cudaMemcpyDeviceToHost,
                                      ctx->stream));
    bool const sync = h_out || h_stats || h_nodes || dpos != positions || dcur != curves;
    return sync ? ctx->check_flags() : AGWN_OK;
}
} // namespace

extern "C" int agwn_param_batch_fractional_bezier3_f64(agwn_context* ctx, const double* positions, int64_t n,
                                                       double* out, const double* x0, const double* curves,
                                                       int64_t n_curves, int min_depth, int max_depth, double tol,
                                                       const uint8_t* start_depth, uint32_t* pair_stats,
                                                       int32_t* nodes_per_query)
{
    return param_entry(ctx, nullptr, 0, 0.f, positions, n, out, x0, curves, n_curves, min_depth, max_depth, tol,
                       start_depth, pair_stats, nodes_per_query);
}

extern "C" int agwn_param_batch_fractional_learned_bezier3_f64(agwn_context* ctx, const agwn_mlp* mlp,
                                                               const double* positions, int64_t n, double* out,
                                                               const double* x0, const double* curves,
                                                               int64_t n_curves, int n_classes, int min_depth,
                                                               int max_depth, double tol, float alpha,
                                                               uint32_t* pair_stats, int32_t* nodes_per_query)
{
    AGWN_CHECK_ARG(mlp, "null network");
    return param_entry(ctx, mlp, n_classes, alpha, positions, n, out, x0, curves, n_curves, min_depth, max_depth, tol,
                       nullptr, pair_stats, nodes_per_query);
}

extern "C" int agwn_param_set_panel_network(agwn_context* ctx, const agwn_mlp* mlp, float beta)
{
    AGWN_CHECK_ARG(ctx, "null context");
    AGWN_CHECK_ARG(beta > 0.f && beta < 1.f, "beta must be in (0, 1)");
    clear_message();
    ctx->panel_mlp = mlp;
    ctx->panel_beta = beta;
    return AGWN_OK;
}

extern "C" int agwn_param_panel_log_bezier3_f64(agwn_context* ctx, const double* positions, int64_t n,
                                                const double* x0, const double* curves, int64_t n_curves,
                                                int min_depth, int max_depth, double tol, uint32_t* log,
                                                int64_t capacity, int64_t* n_entries)
{
    AGWN_CHECK_ARG(ctx && x0 && n_entries && capacity >= 0 && (capacity == 0 || log), "bad arguments");
    AGWN_CHECK_ARG(n >= 0 && n_curves >= 0 && (n == 0 || positions) && (n_curves == 0 || curves), "bad arguments");
    AGWN_CHECK_ARG(n * n_curves < (int64_t(1) << 32), "the log indexes (query, curve) pairs in 32 bits");
    AGWN_CHECK_ARG(min_depth >= 0 && max_depth >= 0 && max_depth <= kParamMaxDepth, "bad depths");
    AGWN_CHECK_ARG(std::isfinite(tol) && tol >= 0, "tol must be finite and >= 0");
    clear_message();
    AGWN_TRY_CUDA(cudaSetDevice(ctx->device));
    *n_entries = 0;
    if (n == 0 || n_curves == 0)
        return AGWN_OK;
    const void *dpos = nullptr, *dcur = nullptr;
    void *dout = nullptr, *dlog = nullptr, *dcnt = nullptr;
    bool h_log = false;
    AGWN_TRY(stage_in(*ctx, positions, sizeof(double) * 3 * n, S_QUERIES, &dpos));
    AGWN_TRY(stage_in(*ctx, curves, sizeof(double) * 12 * n_curves, S_MISC0, &dcur));
    AGWN_TRY(ctx->scratch_reserve(S_OUT, sizeof(double) * n, &dout));
    if (capacity > 0)
        AGWN_TRY(stage_out(*ctx, log, sizeof(uint32_t) * 2 * size_t(capacity), S_MISC2, &dlog, &h_log));
    AGWN_TRY(ctx->scratch_reserve(S_MISC3, sizeof(unsigned long long), &dcnt));
    AGWN_TRY_CUDA(cudaMemsetAsync(dcnt, 0, sizeof(unsigned long long), ctx->stream));
    AGWN_TRY(param_run(*ctx, static_cast<const double*>(dpos), n, static_cast<double*>(dout), x0,
                       static_cast<const double*>(dcur), n_curves, min_depth, max_depth, tol, nullptr, nullptr,
                       nullptr, static_cast<uint32_t*>(dlog), static_cast<unsigned long long*>(dcnt), capacity));
    unsigned long long cnt = 0;
    AGWN_TRY_CUDA(cudaMemcpyAsync(&cnt, dcnt, sizeof(cnt), cudaMemcpyDeviceToHost, ctx->stream));
    AGWN_TRY(ctx->check_flags());
    *n_entries = int64_t(cnt);
    if (h_log)
    {
        int64_t const rows = std::min<int64_t>(int64_t(cnt), capacity);
        AGWN_TRY_CUDA(cudaMemcpyAsync(log, dlog, sizeof(uint32_t) * 2 * size_t(rows), cudaMemcpyDeviceToHost,
                                      ctx->stream));
        AGWN_TRY(ctx->check_flags());
    }
    return AGWN_OK;
}
