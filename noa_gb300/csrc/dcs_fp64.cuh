/*
 * FP64 device functions of the four muon DCS processes.
 *
 *   bremsstrahlung   physics.hh:114-153
 *   pair production  dcs.hh:144-258, 8-node GL numerics.hh:110-129
 *   photonuclear     dcs.hh:261-405, 9-node GL numerics.hh:131-152
 *   ionisation       dcs.hh:408-443
 *
 * Accuracy contract: FP64 -- the reference's own metric (mean relative error,
 * common.hh:228-236) against its CPU output stays below 1e-12.  The formulas
 * are the reference's; what differs is how they are evaluated on a GPU whose
 * FP64 pipe is ~64x slower than its FP32 and integer pipes:
 *
 *  - what depends only on (element, mass) comes precomputed in
 *    noa_dcs_consts (dcs_consts.h), bit-identical to the reference's values;
 *  - log / exp / reciprocal / division inside the quadrature bodies use the
 *    lean64 functions (lean64.cuh): same accuracy class, 0 / 0 / 0 / 1 FP64
 *    instructions instead of CUDA's ~30 / 16 / 8 / 8.5, the rest on the
 *    integer and FP32 pipes; divisions by a shared denominator reuse one
 *    reciprocal;
 *  - what a quadrature node computes between two such functions is 64-bit
 *    fixed-point arithmetic where the pair's ranges allow it (all but extreme
 *    ones; the others take the *_node_wide bodies): 19 and 26 FP64
 *    instructions a node where the FP64 form has 51 and 62.  1e7 pairs:
 *    pair production 5.04 -> 3.29 ms, photonuclear 2.45 -> 1.90 ms, the FP64
 *    pipe at 56% and 46% of its rate (83% and 78%), issue at 62% and 64%;
 *  - branch tests on non-negative doubles compare bit patterns on the
 *    integer pipe (lean64::bits_ge).
 *
 * Every early exit of the reference is decided exactly as the reference
 * decides it: the bound expressions are evaluated in IEEE arithmetic in the
 * reference's order, with __d*_rn intrinsics where the compiler could
 * otherwise fuse a product into an addition.  The zero / non-zero pattern is
 * therefore identical, also for pairs placed exactly on a bound, and NaN
 * inputs propagate as on the CPU.  The `*_live` predicates evaluate only those
 * bounds, so that a kernel can drop closed pairs before the quadrature.
 */
#pragma once

#include "dcs_common.cuh"

namespace noa_dcs {

using lean64::bits_ge;
using lean64::lean_exp;
using lean64::lean_log;
using lean64::lean_rcp;

// Gauss-Legendre literals, numerics.hh:116-121 (8 nodes on [0,1]) and
// numerics.hh:137-144 (9 nodes on [-1,1]).  They are the reference's 8-digit
// truncations; the exact nodes would move results by ~5e-9.
__constant__ double kGL8X[8] = {0.01985507, 0.10166676, 0.2372338, 0.40828268,
                                0.59171732, 0.7627662, 0.89833324, 0.98014493};
__constant__ double kGL8W[8] = {0.05061427, 0.11119052, 0.15685332, 0.18134189,
                                0.18134189, 0.15685332, 0.11119052, 0.05061427};
__constant__ double kGL9X[9] = {0.0000000000000000, -0.8360311073266358, 0.8360311073266358,
                                -0.9681602395076261, 0.9681602395076261, -0.3242534234038089,
                                0.3242534234038089, -0.6133714327005904, 0.6133714327005904};
__constant__ double kGL9W[9] = {0.3302393550012598, 0.1806481606948574, 0.1806481606948574,
                                0.0812743883615744, 0.0812743883615744, 0.3123470770400029,
                                0.3123470770400029, 0.2606106964029354, 0.2606106964029354};

// The nodes in units of 2^-64 and 2^-63, for the fixed-point node bodies.
#define NOA_FX64(x) ((unsigned long long)((x) * 0x1p64))
__constant__ unsigned long long kGL8F[8] = {NOA_FX64(0.01985507), NOA_FX64(0.10166676), NOA_FX64(0.2372338),
                                            NOA_FX64(0.40828268), NOA_FX64(0.59171732), NOA_FX64(0.7627662),
                                            NOA_FX64(0.89833324), NOA_FX64(0.98014493)};
#undef NOA_FX64
#define NOA_FX63(x) ((long long)((x) * 0x1p63))
__constant__ long long kGL9F[9] = {0ll, NOA_FX63(-0.8360311073266358), NOA_FX63(0.8360311073266358),
                                   NOA_FX63(-0.9681602395076261), NOA_FX63(0.9681602395076261),
                                   NOA_FX63(-0.3242534234038089), NOA_FX63(0.3242534234038089),
                                   NOA_FX63(-0.6133714327005904), NOA_FX63(0.6133714327005904)};
#undef NOA_FX63

// Clamp of the reference's `if (v < 0.) v = 0.;` that keeps NaN.
__device__ __forceinline__ double clamp0(double v) {
    const long long b = __double_as_longlong(v);
    return (b < 0 && (b & 0x7FFFFFFFFFFFFFFFLL) <= 0x7FF0000000000000LL) ? 0. : v;
}

// Out-of-line copies of the lean64 functions for the two quadrature bodies.
// Inlined, every call site adds 50 - 100 integer and FP32 instructions, and a
// node with 14 - 22 of them outgrows the instruction cache.  At 1e7 pairs
// the bodies with every function called measure 3.34 / 1.94 ms (pair
// production / photonuclear); the fixed-point logarithm inlined 3.29 / 1.92, the
// fixed-point exponential inlined - / 1.90, both and the reciprocal 3.34 / 1.99.
// So pair production inlines the one and photonuclear the other.
// Bremsstrahlung and ionisation, with a few calls each, inline all.
static __device__ __noinline__ double ol_log(double x) { return lean_log(x); }
static __device__ __noinline__ double ol_exp(double x) { return lean_exp(x); }
static __device__ __noinline__ double ol_rcp(double x) { return lean_rcp(x); }
static __device__ __noinline__ double ol_qdiv(double a, double b) { return lean64::qdiv(a, b); }
static __device__ __noinline__ long long ol_log_fx(double x) { return lean64::lean_log_fx(x); }
static __device__ __noinline__ long long ol_log3p_fx(double x) { return lean64::lean_log3p_fx(x); }
static __device__ __noinline__ long long ol_log_of_fx(long long v) { return lean64::log_of_fx(v); }
static __device__ __noinline__ double ol_exp_fx(long long x) { return lean64::lean_exp_fx(x); }
static __device__ __noinline__ double ol_ratio_fx(unsigned long long n, unsigned long long d) {
    return lean64::ratio_fx(n, d);
}

// Unbiased exponent of a positive double (1024 for inf and NaN).
__device__ __forceinline__ int exponent(double x) { return (__double2hiint(x) >> 20) - 1023; }
__device__ __forceinline__ double twice(double x) {  // normal and finite
    return __hiloint2double(__double2hiint(x) + 0x00100000, __double2loint(x));
}

// Whether E (or K) exceeds q by more than a part in 2^10 - 2^11, both of
// ordinary size (2^-62 to 2^97, and q above 2^-94; NaN and negative values
// fail).  There 1 - q / E and K - q keep 42 bits or more whatever the rounding
// of q / E, so that the quadratures' quotients may be taken lean (their errors
// are no larger for it).  Nearer the edge the reference's own rounding shows in
// the result (by 1 / (1 - q / E) ulp), and its IEEE operations are kept.  High
// words only.
__device__ __forceinline__ bool clear_of_edge(double E, double q) {
    const int he = __double2hiint(E), hq = __double2hiint(q);
    return he >= 0x3C000000 && he < 0x46000000 && hq >= 0x3A000000 && he - hq >= 0x400;
}

// ---------------------------------------------------------------- bremsstrahlung
// q < qe_max decides whether the electron term exists (physics.hh:142):
// cross-multiplied, q (me E + m^2 / 2) < me E^2, and in IEEE arithmetic like
// the reference when the two sides are within 64 ulp.
__device__ __forceinline__ bool brems_below(double E, double q, const noa_dcs_consts &c) {
    const double t = ME * E;
    const long long dist = __double_as_longlong(q * (t + c.br_half_m2)) - __double_as_longlong(t * E);
    if (!(dist >= 64 || dist <= -64) || !clear_of_edge(E, q))
        return brems_below_qe(E, q, c);
    return dist < 0;
}

// The reference's form, for pairs near the kinematic edge (nu -> 1, where its
// rounded nu = q / E shows in 1 - nu) and inputs of unusual size.
__device__ __forceinline__ double brems_reference(double K, double q, const noa_dcs_consts &c) {
    const double mass = c.mass;
    const double sqrte = 1.648721271;
    const double E = K + mass;
    const double nu = __ddiv_rn(q, E);
    const double delta = c.br_half_m2 * lean_rcp(E) * nu * lean_rcp(1. - nu);
    const double Phi_n = clamp0(lean_log(c.br_BZ_n * (mass + delta * c.br_Dn_sqrte_m2) *
                                         lean_rcp(c.br_D_n * (ME + delta * sqrte * c.br_BZ_n))));
    double Phi_e = 0.;
    if (brems_below_qe(E, q, c))
        Phi_e = clamp0(lean_log(c.br_BZe_mass *
                                lean_rcp((1. + delta * c.br_phie_factor) * (ME + delta * sqrte * c.br_BZ_e))));
    const double dcs = c.br_dcs_factor * (c.Zd * Phi_n + Phi_e) * (4. / 3. * (lean_rcp(nu) - 1.) + nu);
    return (dcs < 0.) ? 0. : dcs * c.scale_A;
}

static __device__ __noinline__ double brems_edge(double K, double q, const noa_dcs_consts &c) {
    return brems_reference(K, q, c);
}

// 27 FP64 instructions (42 in the reference's form): the element's factors
// are folded into the two linear forms of each logarithm, and Phi_e is taken as
// the logarithm of the inverse.  nu is q / E rounded to nearest, by Markstein's
// residual correction, as 1 - nu amplifies its last bit towards q = E (with
// q rcp(E) as it is, 1.5 ulp, 1e7 pairs take 499 us against 535, but the mean
// error at 1 - nu in 1e-3 .. 2e-3 is 4.7e-14 against 3.6e-14), and the two scales
// stay two factors, whose product's rounding would be one bias of all of an
// element's results.
__device__ __forceinline__ double brems_fp64(double K, double q, const noa_dcs_consts &c) {
    const double E = K + c.mass;
    if (!clear_of_edge(E, q))
        return brems_edge(K, q, c);
    const double invE = lean_rcp(E);
    const double nu0 = q * invE;
    const double nu = fma(fma(-nu0, E, q), invE, nu0);
    const double delta = c.br_half_m2 * invE * nu * lean_rcp(1. - nu);
    const double Phi_n = clamp0(lean_log(fma(delta, c.br_n1, c.br_n0) * lean_rcp(fma(delta, c.br_d1, c.br_d0))));
    double Phi_e = 0.;
    if (brems_below(E, q, c))
        Phi_e = clamp0(-lean_log(fma(delta, c.br_e1, c.br_e0) * fma(delta, c.br_f1, ME)));
    const double shape = fma(4. / 3., lean_rcp(nu), nu - 4. / 3.);
    return clamp0(c.br_dcs_factor * fma(c.Zd, Phi_n, Phi_e) * shape) * c.scale_A;
}

// ---------------------------------------------------------------- pair production
// The rare part of pprod_live, out of line so that the kernels that inline
// pprod_live once per item keep one copy of it: the float-float argmin
// (~1e-13 relative here), whose distance from 1 decides beyond 1e-10, and
// the IEEE argmin near q = 4 me (1 - x0 < 1e-4, where 1 - x0 amplifies the
// error of x0), for extreme K, or within 1e-10.  Scalars only (a reference
// to the constants would copy them to local memory).
static __device__ __noinline__ bool pprod_live_tail(double K, double q, double mass, float inv_mass_h, float inv_mass_l,
                                             float x0) {
    noa_dcs_consts c;  // pprod_argmin_ff / _exact read only these three fields
    c.mass = mass;
    c.inv_mass_h = inv_mass_h;
    c.inv_mass_l = inv_mass_l;
    if (x0 < 0.9999f && fpconv::f32(K) < 1e15f) {
        const FF am = pprod_argmin_ff(K, q, c);
        const float d = (am.h - 1.f) + am.l;  // am.h - 1 is exact for am.h in [0.5, 2]
        if (am.h >= 0.5f && am.h <= 2.f && fabsf(d) > 1e-10f)
            return d < 0.f;
        if (am.h > 1e-30f && am.h < 0.5f)
            return true;
        if (am.h > 2.f && am.h < 1e30f)
            return false;
    }
    const double am = pprod_argmin_exact(K, q, c);
    return !((am >= 1.) || (am <= 0.));
}

// The whole open / closed decision in the reference's IEEE arithmetic
// (dcs.hh:151-156 and the argmin check), out of line: reached only where float
// cannot decide, so that the inlined fast path carries no FP64 comparison
// (the compiler would otherwise evaluate the short exact tests
// unconditionally, as predicated FP64 instructions, for every pair).
static __device__ __noinline__ bool pprod_live_exact(double K, double q, double mass, double shift,
                                                     float inv_mass_h, float inv_mass_l) {
    if (q <= 4. * ME)
        return false;
    if (q >= K + shift)
        return false;
    return pprod_live_tail(K, q, mass, inv_mass_h, inv_mass_l, 1.f);
}

__device__ __forceinline__ bool pprod_live(double K, double q, const noa_dcs_consts &c) {
    // NaN outside the normal float range: the range test below fails there
    const float Kf = fpconv::f32_normal(K), qf = fpconv::f32_normal(q);
    if (!(Kf > 1e-20f && Kf < 1e30f && qf > 1e-20f && qf < 1e30f))  // outside the float-safe range (and NaN)
        return pprod_live_exact(K, q, c.mass, c.pp_kmax_shift, c.inv_mass_h, c.inv_mass_l);
    // q <= 4 me and q >= K + m (1 - 0.75 sqrt(e) Z^1/3) (dcs.hh:151-156) in
    // float, with the IEEE comparison within a relative margin of 1e-5
    constexpr float four_me = (float)(4. * ME);
    if (qf < four_me * 0.99999f)
        return false;
    const float shift = c.pp_kmax_shift_f;
    const float ub = Kf + shift, margin = 1e-5f * (Kf + fabsf(shift));
    if (qf >= ub + margin)
        return false;
    if (!(qf > four_me * 1.00001f) || !(qf <= ub - margin))
        return pprod_live_exact(K, q, c.mass, c.pp_kmax_shift, c.inv_mass_h, c.inv_mass_l);
    // argmin in float, with K - q (gamma - q/m = 1 + (K - q)/m) as a
    // float-float difference; the reference's IEEE value decides only within
    // 1e-5 of a bound
    const FF kmq = ff_add(ff_split(K), ff_neg(ff_split(q)));
    const float im = c.inv_mass_h;
    const float x0 = four_me * lean64::rcp_approx(qf);
    const float gamma = 1.f + Kf * im;
    const float x1 = 6.f * lean64::rcp_approx(gamma * (1.f + (kmq.h + kmq.l) * im));
    const float a = (x0 + 2.f * (1.f - x0) * x1) * lean64::rcp_approx(1.f + (1.f - x1) * sqrtf(fmaxf(1.f - x0, 0.f)));
    if (fabsf(a - 1.f) > 1e-5f && a > 1e-30f && a < 1e30f && x0 < 0.9f)
        return a < 1.f;
    return pprod_live_tail(K, q, c.mass, c.inv_mass_h, c.inv_mass_l, x0);
}

// beta = nu^2 / (2 (1 - nu)) and argmin with the reference's own rounding
// (nu = q / E rounded, argmin in IEEE order), for pairs near an edge: 1 - nu
// and log(argmin) amplify the last bit there.
static __device__ __noinline__ double2 pprod_edge(double K, double q, double mass) {
    noa_dcs_consts c;  // pprod_argmin_exact reads only the mass
    c.mass = mass;
    const double nu = __ddiv_rn(q, K + mass);
    return make_double2(0.5 * nu * nu * ol_rcp(1. - nu), pprod_argmin_exact(K, q, c));
}

// What one open pair's nodes share.  With s = 1 - rho^2 = eps (2 - eps) every
// factor of the reference's integrand that does not take a logarithm is linear
// in s (dcs.hh:188-216):
//   (2 + rho^2)(1 + beta) + xi (3 + rho^2) = a0 + s (a1 - xi),  xi = xf s
//   rho^2 + 2 beta (2 - rho^2)             = pd - 2 s hd
//   (1 + rho^2)(1 + 1.5 beta) - (1 + 2 beta) s / xi = m0 + s m1
//   xi / 2 (5 - rho^2 + beta (3 + rho^2))  = xi (b0 + s b1)
// c1 = 2 sqrt(e) me / q, times xf, scales the screening lengths.  In fixed
// point t = -tmin and beta = B 2^(h - 60), h >= 0 the least that keeps B below
// 2^60; h < 0 marks a pair whose nodes are pprod_node_wide's (cx is then c1).
struct PprodPair {
    double tmin, xf, beta, a0, a1, pd, hd, m0, m1, b0, b1, cx;
    long long t, B, h;
};

// The nodes of a pair outside the fixed-point ranges, in FP64 throughout: 6
// logarithms, an exponential and 6 reciprocals.
static __device__ __noinline__ double pprod_node_wide(double tmin, double xf, double beta, double c1, int j,
                                                      const noa_dcs_consts &c);

__device__ __forceinline__ void pprod_setup(double K, double q, const noa_dcs_consts &c, PprodPair &p) {
    const double E = K + c.mass;
    const double rq = ol_rcp(q);
    double beta, argmin;
    bool edge = !clear_of_edge(K, q);
    if (!edge) {
        // gamma = E / m and gamma - q / m = (E - q) / m
        const double rEE = ol_rcp(E * (E - q));
        beta = (0.5 * q) * q * rEE;
        const double x0 = 4. * ME * rq, x1 = c.pp_6m2 * rEE;
        const double omx0 = 1. - x0;
        argmin = fma(2., omx0 * x1, x0) * ol_rcp(fma(1. - x1, lean64::lean_sqrt(omx0), 1.));
        edge = __double2hiint(argmin) >= 0x3FEFF800;  // argmin >= 1 - 2^-10
    }
    if (edge) {
        const double2 e = pprod_edge(K, q, c.mass);
        beta = e.x;
        argmin = e.y;
    }
    p.tmin = ol_log(argmin);
    p.beta = beta;
    p.xf = c.pp_half_r2 * beta;
    p.a0 = fma(3., beta, 3.);
    p.a1 = fma(4., p.xf, -1. - beta);
    p.pd = fma(2., beta, 1.);
    p.hd = 0.5 - beta;
    p.m0 = fma(-p.pd, ol_rcp(p.xf), fma(3., beta, 2.));
    p.m1 = fma(-1.5, beta, -1.);
    p.b0 = fma(2., beta, 2.);
    p.b1 = fma(-0.5, beta, 0.5);
    const double c1 = c.pp_2sm * rq;
    // argmin <= s <= 1: every logarithm of the node body stays below 64
    const int eb = exponent(beta), ex = exponent(p.xf), ea = exponent(argmin);
    const bool fits = eb > -1000 && eb < 50 && ex > -1000 && ex < 50 && ea < 0 && ea >= -50 && ex + ea >= -85 &&
                      c.pp_log_kappa_fx != INT64_MIN;
    const int h = eb < 0 ? 0 : eb + 1;
    p.cx = fits ? c1 * p.xf : c1;
    p.t = lean64::to_fx(-p.tmin, 57);
    p.B = lean64::to_fx(beta, 60 - h);
    p.h = fits ? h : -1;
}

// Clamp of the reference's `if (Phi < 0.) Phi = 0.;` for -Phi; keeps NaN.
__device__ __forceinline__ double clamp0_neg(double v) {
    return (unsigned long long)__double_as_longlong(v) - 1ull < 0x7FF0000000000000ULL ? 0. : v;
}

// Node j: -(1 - rho) (Phi_e + Phi_mu / r^2), 19 FP64 instructions (about 75
// in the reference's form) beside 7 logarithms, an exponential and 6
// reciprocals.  The screening logarithms are those of the inverse arguments,
//   Le  = -(log d + log(1 / xe + cLe) / 2),   d = 1 / AZ13 + c1 xe / s
//   Lmu = -(log(1 / AZ13 + c1 xmu / s) + log kappa),
// which spares their products with 1 / d and the square root.  Ye and Ymu
// (dcs.hh:196-216), quotients of sums of products of s, beta and a logarithm,
// are 64-bit integers up to the quotient, 1 + Y = (N + D) / D:
//   Ye:  N = 4 + 8 beta + s (1 - 4 beta),  D = (2 + 6 beta) log(3 + 1 / xi) + s (1 - 2 beta) - (1 + 2 beta)
//   Ymu: N = 5 + 6 beta - s (1 + 3 beta),  D = (3 + 4 beta - s (3/2 + 2 beta)) log(3 + xi) + (3 s - 1) / 2
// D stays above a third of 1 + beta, so that units of 2^-53 (1 + beta) suffice.
// The arguments 1 + xi and 1 + 1 / xi keep the reference's rounding to double,
// which the cancellation in Phi near xi = 10^3 makes visible.
// The reference's two forms of each Phi (xi above 10^3, below 10^-3) differ in
// operands only: selects, not two branches that nearly every warp would both take.
__device__ __forceinline__ double pprod_node(const PprodPair &p, int j, const noa_dcs_consts &c) {
    if (p.h < 0)
        return pprod_node_wide(p.tmin, p.xf, p.beta, p.cx, j, c);
    const double eps = ol_exp_fx(-(long long)lean64::detail::mulhi_u64((unsigned long long)p.t, kGL8F[j]));
    const double s = fma(-eps, eps, twice(eps));
    const double xi = p.xf * s;
    const double xi_i = ol_rcp(xi);
    const double opxi = 1. + xi;
    const double inv_opxi = ol_rcp(opxi);
    const double crs = p.cx * xi_i;

    // units of 2^(h - 60): u = 1, s and s beta; D and N in units of 2^(h - 53)
    const int h = (int)p.h;
    const long long B = p.B, u = (long long)((1ull << 60) >> h);
    const unsigned long long sf = lean64::unit_to_fx62(s);
    const long long su = (long long)(sf >> (h + 2)), sB = lean64::fx_mul((long long)sf, B, 62);
    const auto times_log = [](long long a, long long l) {
        return (long long)lean64::detail::mulhi_u64((unsigned long long)a, (unsigned long long)l);
    };
    const long long De = times_log(2 * u + 6 * B, ol_log3p_fx(xi_i)) + ((su - 2 * sB - u - 2 * B) >> 7);
    const long long Ne = ((u + 2 * B) >> 5) + ((su - 4 * sB) >> 7);
    const double xe = opxi * ol_ratio_fx((unsigned long long)(Ne + De), (unsigned long long)De);
    const long long Dm = times_log(3 * u + 4 * B - su - (su >> 1) - 2 * sB, ol_log3p_fx(xi)) + ((3 * su - u) >> 8);
    const long long Nm = ((5 * (u >> 1) + 3 * B) >> 6) - ((su + 3 * sB) >> 7);
    const double xmu = opxi * ol_ratio_fx((unsigned long long)(Nm + Dm), (unsigned long long)Dm);
    // (s - beta) / (1 + xi) + s - 4 and (s - beta) xi / (1 + xi) + (1 + 2 beta) s
    const long long inv = (long long)lean64::unit_to_fx62(inv_opxi);
    const double Ce = lean64::from_fx_any(lean64::fx_mul(inv, su - B, 62) + su - 4 * u, 60 - h);
    const double Cm = lean64::from_fx_any(lean64::fx_mul((1ll << 62) - inv, su - B, 62) + su + 2 * sB, 60 - h);

    const bool far = bits_ge(xi, 1E+03), near = !bits_ge(xi, 1.0000000000000002E-03);  // xi <= 1e-3
    const double Be = fma(fma(s, far ? p.hd : p.a1 - xi, far ? p.pd : p.a0), far ? xi_i : ol_log(1. + xi_i), far ? 0. : Ce);
    const long long le = lean64::lean_log_fx(fma(crs, xe, c.pp_inv_AZ13)) + (lean64::lean_log_fx(ol_rcp(xe) + c.pp_cLe) >> 1);
    const double Pe = clamp0_neg(Be * lean64::from_fx_any(le));
    const double Bmu = fma(fma(s, near ? p.b1 : p.m1, near ? p.b0 : p.m0), near ? xi : ol_log(opxi), near ? 0. : Cm);
    const long long lm = lean64::lean_log_fx(fma(crs, xmu, c.pp_inv_AZ13)) + c.pp_log_kappa_fx;
    const double Pmu = clamp0_neg(Bmu * lean64::from_fx_any(lm));
    // 1 - rho as the reference rounds it: for small eps its last bit (2^-54 / eps) shows in the result
    return fma(Pmu, c.pp_inv_r2, Pe) * lean64::round_by_one(eps);
}

static __device__ __noinline__ double pprod_node_wide(double tmin, double xf, double beta, double c1, int j,
                                                      const noa_dcs_consts &c) {
    const double eps = ol_exp(kGL8X[j] * tmin);
    const double s = eps * (2. - eps);
    const double xi = xf * s;
    const double xi_i = ol_rcp(xi);
    const double opxi = 1. + xi;
    const double inv_opxi = ol_rcp(opxi);
    const double sb = s - beta;
    const double crs = c1 * ol_rcp(s);
    const double dc = fma(-2., beta, -1.), ds = fma(-2., beta, 1.);

    double Be;
    if (bits_ge(xi, 1E+03))
        Be = xi_i * fma(0.5 * s, ds, -dc);
    else
        Be = fma(fma(s, fma(-s, xf, fma(4., xf, -1. - beta)), fma(3., beta, 3.)), ol_log(1. + xi_i),
                 fma(sb, inv_opxi, s - 4.));
    const double Ye = fma(s, fma(-4., beta, 1.), fma(8., beta, 4.)) *
                      ol_rcp(fma(fma(6., beta, 2.), ol_log(3. + xi_i), fma(s, ds, dc)));
    const double xe = fma(opxi, Ye, opxi);
    const double de = fma(crs, xe, c.pp_inv_AZ13);
    const double Pe = clamp0_neg(Be * ol_log(de * de * (ol_rcp(xe) + c.pp_cLe)));

    double Bmu;
    if (!bits_ge(xi, 1.0000000000000002E-03))  // xi <= 1e-3
        Bmu = 0.5 * xi * fma(beta, 4. - s, 4. + s);
    else
        Bmu = fma(fma(s, fma(-1.5, beta, -1.), fma(dc, ol_rcp(xf), fma(3., beta, 2.))), ol_log(opxi),
                  fma(sb, xi * inv_opxi, -dc * s));
    const double Ymu = fma(s, fma(-3., beta, -1.), fma(6., beta, 5.)) *
                       ol_rcp(fma(fma(s, fma(-2., beta, -1.5), fma(4., beta, 3.)), ol_log(3. + xi), fma(1.5, s, -0.5)));
    const double xmu = fma(opxi, Ymu, opxi);
    const double Pmu = clamp0_neg(Bmu * ol_log(c.pp_kappa * fma(crs, xmu, c.pp_inv_AZ13)));
    return fma(Pmu, c.pp_inv_r2, 0.5 * Pe) * (1. - (1. - eps));
}

// From the sum of the nodes: the atomic-electron form factor zeta and the
// scales.  (mass + K) / E of the reference's two factors cancels.
__device__ __forceinline__ double pprod_finish(double K, double q, double tmin, double sum, const noa_dcs_consts &c) {
    const double E = K + c.mass;
    const double gamma = E * c.inv_mass;
    double zeta = 0.;
    if (!(gamma <= 35.)) {
        zeta = 0.073 * ol_log(gamma * ol_rcp(fma(c.pp_g1, gamma, 1.))) - 0.26;
        if (zeta <= 0.)
            zeta = 0.;
        else
            zeta = zeta * ol_rcp(0.058 * ol_log(gamma * ol_rcp(fma(c.pp_g2, gamma, 1.))) - 0.14);
    }
    return clamp0(c.pp_cZs * (c.Zd + zeta) * (E - q) * (tmin * sum) * ol_rcp(q));
}

// An open pair (pprod_live), its nodes one after the other.
__device__ __forceinline__ double pprod_fp64(double K, double q, const noa_dcs_consts &c) {
    PprodPair p;
    pprod_setup(K, q, c, p);
    double sum = 0.;
#pragma unroll 1  // rolled: smaller code, same FP64 work
    for (int j = 0; j < 8; j++)
        sum = fma(kGL8W[j], pprod_node(p, j, c), sum);
    return pprod_finish(K, q, p.tmin, sum, c);
}

// ---------------------------------------------------------------- photonuclear
// Q2min and Q2max with the reference's own rounding, for pairs near an edge.
static __device__ __noinline__ double2 photo_edge(double K, double q, double mass) {
    const double y = __ddiv_rn(q, K + mass);
    return make_double2(__ddiv_rn(x_mul(x_mul(x_mul(mass, mass), y), y), x_sub(1., y)),
                        x_sub(x_mul(2.0 * PH_M, q - PH_MPI), PH_MPI * PH_MPI));
}

// photo_window's open / closed decision (dcs.hh:357-381), float first: in
// float every bound is decided with a relative margin of 1e-5 (1e-4 of the
// terms for Q2max >= Q2min, whose float difference cancels near q_min; with
// q_min = mpi (1 + mpi / 2M), Q2max = 2M (q - q_min) exactly in real
// arithmetic), far above float rounding; pairs within a margin, and inputs
// outside the float-safe range (zero, NaN, inf, huge), take the exact IEEE
// check.  Only the closed / open answer is taken from float, never a value.
__device__ __forceinline__ bool photo_live(double K, double q, const noa_dcs_consts &c) {
    // NaN outside the normal float range: the range test below fails there
    const float Kf = fpconv::f32_normal(K), qf = fpconv::f32_normal(q);
    if (Kf >= 1e-30f && Kf <= 1e30f && qf >= 1e-30f && qf <= 1e30f) {
        constexpr float lo = 0.99999f, hi = 1.00001f;
        const float qmin = c.ph_q_min_f, cut = 2E-03f * Kf;
        if (qf < lo || qf < cut * lo || qf > Kf * hi || qf < qmin * lo)
            return false;  // q < 1, q < 2e-3 K, q >= E - m (= K to an ulp), q <= q_min
        if (!(qf < hi || qf < cut * hi || qf > Kf * lo || qf < qmin * hi)) {
            const float m = c.mass_h;
            const float Ef = Kf + m, Emq = fpconv::f32_normal(K + c.mass - q);  // q < K (1 - 1e-5): no cancellation
            const float y = qf / Ef, omy = Emq / Ef;
            const float Q2min = m * m * y * y / omy;
            const float Q2max = (float)(2.0 * PH_M) * (qf - qmin);
            const float margin = 1e-4f * ((float)(2.0 * PH_M) * qf + Q2min);
            if (Q2max < Q2min - margin)
                return false;
            if (Q2max > Q2min + margin)
                return true;
        }
    }
    double a, b;
    return photo_window(K, q, c, a, b);
}

// What one open pair's nodes share, in fixed point (units of 2^-57) but for
// hd, h and what enters the last factor.  A pair outside the fixed-point ranges
// has `wide` set and pc and k2 as doubles (bits), and is evaluated by photo_node_wide.
struct PhotoPair {
    double hd;              // log Q2 = pc + hd x_j
    double h;               // x = h Q2
    double omy, yy, invEE;  // 1 - y, y^2, 1 / E^2
    long long pc, hdf;      // log Q2's, hdf in units of 2^-58
    long long lP, lR;       // -log(mP2 + 2 M q), -log(mR2 + 2 M q)
    long long k2;           // DRSS exponent k1 log Q2 + k2
    long long wide;
};

// The nodes of a pair outside the fixed-point ranges, in FP64 throughout: 6
// logarithms, 10 exponentials and 8 reciprocals.
static __device__ __noinline__ double photo_node_wide(const double pc, const double hd, const double h,
                                                      const double k2, const double omy, const double yy,
                                                      const double invEE, int j, const noa_dcs_consts &c);

__device__ __forceinline__ void photo_setup(double K, double q, const noa_dcs_consts &c, PhotoPair &p) {
    const double E = K + c.mass;
    const double invE = ol_rcp(E);
    double Q2min = 0., Q2max = 0.;
    bool edge = !clear_of_edge(K, q);
    if (!edge) {
        const double mq = c.mass * q;
        Q2min = mq * mq * ol_rcp(E * (E - q));
        Q2max = fma(2.0 * PH_M, q, -(2.0 * PH_M * PH_MPI + PH_MPI * PH_MPI));
        edge = __double2hiint(Q2max) - __double2hiint(Q2min) < 0x400;  // a nearly closed window
    }
    if (edge) {
        const double2 e = photo_edge(K, q, c.mass);
        Q2min = e.x;
        Q2max = e.y;
    }
    const double half_min = 0.5 * ol_log(Q2min), log_max = ol_log(Q2max);
    const double pc = fma(0.5, log_max, half_min);
    p.hd = fma(0.5, log_max, -half_min);
    p.h = (0.5 / PH_M) * ol_rcp(q);
    const double k2 = fma(c.ph_k1, ol_log(p.h), c.ph_k0);
    const double y = q * invE;
    p.omy = (E - q) * invE;
    p.yy = y * y;
    p.invEE = invE * invE;
    // 2^-26 <= Q2 < 2^41 and a window of a factor above 2 (its nodes keep 1 - x
    // above 0.01) hold every exponent within (-64, 64) and every exponential
    // that is added within 64; |DRSS exponent| < 8
    const bool fits = exponent(Q2min) >= -26 && exponent(Q2max) < 41 && exponent(Q2max) - exponent(Q2min) >= 2 &&
                      exponent(fabs(k2)) < 2 && exponent(fabs(c.ph_k1)) < 0;
    p.wide = fits ? 0 : 1;
    p.pc = fits ? lean64::to_fx(pc, 57) : __double_as_longlong(pc);
    p.k2 = fits ? lean64::to_fx(k2, 57) : __double_as_longlong(k2);
    p.hdf = lean64::to_fx(p.hd, 58);
    p.lP = (long long)(0ull - (unsigned long long)ol_log_fx(fma(2.0 * PH_M, q, 49.457)));
    p.lR = (long long)(0ull - (unsigned long long)ol_log_fx(fma(2.0 * PH_M, q, 0.15052)));
}

// Node j: (F2A / (A / 2)) Q2 dds of dcs.hh:289-354, 26 FP64 instructions
// (about 90 in the reference's form) beside 7 logarithms, 9 exponentials and 6
// reciprocals; what the ALLM fit and the DRSS shadowing put between these is
// 64-bit integer arithmetic.  W2 - M2 = Q2 (1/x - 1) = 2 M q - Q2, which makes the
// denominators of xP and xR constants of the pair; log x and log(Q2 / 0.04)
// follow from log Q2 = pc + hd x_j; c1 + (c1 - c2) (1 / (1 + e) - 1) is
// c2 + (c1 - c2) / (1 + e); Q2 / (Q2 + m02) and the shadowing factor are
// exponents of F2's two terms; Q2 / Q2^2 is taken together.
__device__ __forceinline__ double photo_node(const PhotoPair &p, int j, const noa_dcs_consts &c) {
    if (p.wide)
        return photo_node_wide(__longlong_as_double(p.pc), p.hd, p.h, __longlong_as_double(p.k2), p.omy, p.yy, p.invEE,
                               j, c);
    using lean64::fx_const;
    using lean64::fx_mul;
    // ALLM parameters, dcs.hh:262-288.
    const double m02 = 0.31985, mP2 = 49.457, mR2 = 0.15052, Q02 = 0.52544;

    const long long lq = p.pc + lean64::detail::mulhi_s64(p.hdf, kGL9F[j]);
    const double Q2 = ol_exp_fx(lq);
    const double invQ2 = ol_rcp(Q2);
    const double x = p.h * Q2;
    // ALLM F2, dcs.hh:289-306: t = log((Q2 + Q02) / Lambda2) / log(Q02 / Lambda2), lnt = log(log t)
    const long long log_inv_lambda2 = 393322452271277762ll;  // log(1 / 0.06527)
    const long long log_inv_log_q02 = -105939969078771798ll;  // -log(log(0.52544 / 0.06527))
    const long long lnt = ol_log_of_fx(ol_log_of_fx(ol_log_fx(Q2 + Q02) + log_inv_lambda2) + log_inv_log_q02);
    const auto power = [lnt](double a) { return lean64::exp_to_fx(fx_mul(lnt, fx_const(a))); };
    // 1 / (1 + e) in units of 2^-62 (of 2^lz / (1 + e), shifted back)
    const auto inv_1p = [](long long e) {
        const unsigned long long d = (unsigned long long)(e + fx_const(1.));
        const int lz = lean64::detail::clz64(d);  // 1 <= d 2^-57 < 64
        return (long long)(lean64::rcp_wide(d << lz) >> (6 - lz));
    };
    const long long cP =
        fx_const(0.22291) + lean64::detail::mulhi_s64(inv_1p(power(2.1979)), fx_const(0.28067 - 0.22291, 59));
    const long long aP =
        fx_const(-0.44812) + lean64::detail::mulhi_s64(inv_1p(power(1.1709)), fx_const(-0.0808 + 0.44812, 59));
    const long long bP = fx_const(0.36292) + fx_mul(power(1.8439), fx_const(1.8917));
    const long long cR = fx_const(0.80107) + fx_mul(power(3.4942), fx_const(0.97307));
    const long long aR = fx_const(0.58400) + fx_mul(power(2.6063), fx_const(0.37888));
    const long long bR = fx_const(0.01147) + fx_mul(power(0.49338), fx_const(3.7582));
    const long long l1x = ol_log_fx(1. - x);
    // Q2 / (Q2 + m02) and the DRSS shadowing, dcs.hh:310-319
    long long f = lq - ol_log_fx(Q2 + m02);
    if (!bits_ge(x, 0.04))
        f += bits_ge(x, 0.0014) ? fx_mul(lq, c.ph_k1_fx) + p.k2 : c.ph_log_a_low_fx;
    double F2 = lean64::from_fx(cP) * ol_exp_fx(fx_mul(aP, ol_log_fx(Q2 + mP2) + p.lP) + fx_mul(bP, l1x) + f);
    F2 = fma(lean64::from_fx(cR), ol_exp_fx(fx_mul(aR, ol_log_fx(Q2 + mR2) + p.lR) + fx_mul(bR, l1x) + f), F2);
    // 2 - 1.85 x + 2.45 x^2 - 2.35 x^3 + x^4, in units of 2^-61
    const long long xf = (long long)lean64::unit_to_fx62(x);
    const auto times_x = [xf](long long a) { return lean64::detail::mulhi_s64(xf, a) * 4; };
    const long long poly =
        fx_const(2., 61) + times_x(fx_const(-1.85, 61) +
                                   times_x(fx_const(2.45, 61) + times_x((xf >> 1) - fx_const(2.35, 61))));
    F2 *= lean64::from_fx(poly, 61);
    // 1 + R, Whitlow, dcs.hh:322-332
    const bool low = !bits_ge(Q2, 0.3);
    const double q2 = low ? 0.3 : Q2;
    const double inv_q2 = low ? 1. / 0.3 : invQ2;
    const long long lg = low ? 290378127760058573ll : lq + 463888894893706459ll;  // log(25 q2)
    const double theta = fma(12.0 * 0.015625 * q2, ol_rcp((1.0 + q2) * fma(x, x, 0.015625)), 1.);
    const double R1 = fma(-0.3534, ol_rcp(fma(q2, q2, 0.09)),
                          fma(0.5747, inv_q2,
                              fma(theta, ol_ratio_fx((unsigned long long)fx_const(0.635), (unsigned long long)lg), 1.)));
    // dcs.hh:348-354, times Q2
    const double t = fma(-c.ph_m2, invQ2, 0.5) * fma(Q2, p.invEE, p.yy);
    const double dds = fma(fma(t, ol_rcp(R1), p.omy), invQ2, -0.25 * p.invEE);
    return F2 * dds;
}

static __device__ __noinline__ double photo_node_wide(const double pc, const double hd, const double h,
                                                      const double k2, const double omy, const double yy,
                                                      const double invEE, int j, const noa_dcs_consts &c) {
    // ALLM parameters, dcs.hh:262-288.
    const double m02 = 0.31985, mP2 = 49.457, mR2 = 0.15052, Q02 = 0.52544;
    const double cP1 = 0.28067, cP2 = 0.22291, cP3 = 2.1979;
    const double aP1 = -0.0808, aP2 = -0.44812, aP3 = 1.1709;
    const double bP1 = 0.36292, bP2 = 1.8917, bP3 = 1.8439;
    const double cR1 = 0.80107, cR2 = 0.97307, cR3 = 3.4942;
    const double aR1 = 0.58400, aR2 = 0.37888, aR3 = 2.6063;
    const double bR1 = 0.01147, bR2 = 3.7582, bR3 = 0.49338;
    const double inv_lambda2 = 1. / 0.06527;

    const double two_Mq = ol_rcp(h);
    const double inv_dP = ol_rcp(two_Mq + mP2), inv_dR = ol_rcp(two_Mq + mR2);
    const double lq = fma(hd, kGL9X[j], pc);
    const double Q2 = ol_exp(lq);
    const double invQ2 = ol_rcp(Q2);
    const double x = h * Q2;
    // ALLM F2, dcs.hh:289-306
    const double lnt = ol_log(ol_log(ol_log((Q2 + Q02) * inv_lambda2) * c.ph_inv_log_q02));
    const double cP = fma(cP1 - cP2, ol_rcp(1.0 + ol_exp(cP3 * lnt)), cP2);
    const double aP = fma(aP1 - aP2, ol_rcp(1.0 + ol_exp(aP3 * lnt)), aP2);
    const double bP = fma(bP2, ol_exp(bP3 * lnt), bP1);
    const double l1x = ol_log(1. - x);
    double F2 = cP * ol_exp(fma(aP, ol_log((Q2 + mP2) * inv_dP), bP * l1x));
    const double cR = fma(cR2, ol_exp(cR3 * lnt), cR1);
    const double aR = fma(aR2, ol_exp(aR3 * lnt), aR1);
    const double bR = fma(bR2, ol_exp(bR3 * lnt), bR1);
    F2 = fma(cR, ol_exp(fma(aR, ol_log((Q2 + mR2) * inv_dR), bR * l1x)), F2);
    F2 = Q2 * ol_rcp(Q2 + m02) * F2;
    // DRSS shadowing, dcs.hh:310-319
    if (!bits_ge(x, 0.0014))
        F2 *= c.ph_a_low;
    else if (!bits_ge(x, 0.04))
        F2 *= ol_exp(fma(c.ph_k1, lq, k2));
    F2 *= fma(x, fma(x, fma(x, x - 2.35, 2.45), -1.85), 2.0);
    // 1 + R, Whitlow, dcs.hh:322-332
    const bool low = !bits_ge(Q2, 0.3);
    const double q2 = low ? 0.3 : Q2;
    const double inv_q2 = low ? 1. / 0.3 : invQ2;
    const double lg = low ? 2.0149030205422647 : lq + 3.2188758248682006;  // log(25 q2)
    const double theta = fma(12.0 * 0.015625 * q2, ol_rcp((1.0 + q2) * fma(x, x, 0.015625)), 1.);
    const double R1 = fma(-0.3534, ol_rcp(fma(q2, q2, 0.09)),
                          fma(0.5747, inv_q2, fma(0.635 * theta, ol_rcp(lg), 1.)));
    // dcs.hh:348-354, times Q2
    const double t = fma(-c.ph_m2, invQ2, 0.5) * fma(Q2, invEE, yy);
    const double dds = fma(fma(t, ol_rcp(R1), omy), invQ2, -0.25 * invEE);
    return F2 * dds;
}

__device__ __forceinline__ double photo_finish(double K, double q, double hd, double sum, const noa_dcs_consts &c) {
    // E / q first: E times the rest overflows for K above 1e245, where the value does not
    return clamp0(c.ph_scale_A * sum * hd * ((K + c.mass) * ol_rcp(q)));
}

// An open pair (photo_live), its nodes one after the other.
__device__ __forceinline__ double photo_fp64(double K, double q, const noa_dcs_consts &c) {
    PhotoPair p;
    photo_setup(K, q, c, p);
    double sum = 0.;
#pragma unroll 1
    for (int j = 0; j < 9; j++)
        sum = fma(kGL9W[j], photo_node(p, j, c), sum);
    return photo_finish(K, q, p.hd, sum, c);
}

// ---------------------------------------------------------------- ionisation
// ionisation's first exit (dcs.hh:413-419: W_max < 5% K or q > W_max),
// decided in float first: W_max = 2 me K (K + 2 mass) / ((mass + me)^2 +
// 2 me K) has only positive terms, so its float value is within a few float
// ulps; each bound is decided with a relative margin of 1e-5.  1: the exit is
// not taken, 0: it is taken, -1: within a margin or outside the float-safe
// range (zero, NaN, inf, huge), where the caller takes the exact IEEE test.
// Only the decision is taken from float, never a value.
__device__ __forceinline__ int ion_first_exit(double K, double q, const noa_dcs_consts &c) {
    const float Kf = fpconv::f32_normal(K), qf = fpconv::f32_normal(q);  // NaN outside the normal range
    if (!(Kf >= 1e-30f && Kf <= 1e15f && qf >= 1e-30f && qf <= 1e30f))
        return -1;
    constexpr float me = (float)NOA_ELECTRON_MASS;
    const float W = 2.f * me * Kf * (Kf + 2.f * c.mass_h) / (c.io_cm_h + 2.f * me * Kf);
    constexpr float lo = 0.99999f, hi = 1.00001f;
    const float cut = (float)NOA_X_FRACTION * Kf;
    if (W < cut * lo || qf > W * hi)
        return 0;
    return (W > cut * hi && qf < W * lo) ? 1 : -1;
}

// 22 FP64 instructions on the open path (about 35 in the reference's form):
// 1 / W_max = (E + cW) / P2, and 1 / P2 is taken out of the close-collision
// bracket; the comparisons are of bit patterns where K and q are positive and
// normal (first > 0).
__device__ __forceinline__ double ion_fp64(double K, double q, const noa_dcs_consts &c) {
    const double E = K + c.mass;
    const double P2 = K * (E + c.mass);
    const int first = ion_first_exit(K, q, c);
    if (first == 0)
        return 0.;
    double EcW = E + c.io_cW;  // P2 / W_max
    bool radiative;
    if (first < 0) {
        const double P2_ref = K * (K + 2. * c.mass);
        const double Wmax = ion_wmax(P2_ref, E, c);
        if ((Wmax < NOA_X_FRACTION * K) || (q > Wmax) || (q <= c.io_Wmin))
            return 0.;
        EcW = P2 * lean_rcp(Wmax);
        radiative = K >= c.io_k_rad;
    } else {
        if (bits_ge(c.io_Wmin, q))
            return 0.;
        radiative = bits_ge(K, c.io_k_rad);
    }
    const double inv_q = lean_rcp(q);
    const double cs = c.io_cZA * E * lean_rcp(P2) * fma(inv_q, fma(E * E, inv_q, -EcW), 0.5);
    if (!radiative)
        return cs;
    const double L1 = lean_log(fma(q, 2. / ME, 1.));
    return cs * fma(1.16141E-03 * L1, lean_log(c.io_4_inv_m2 * E * (E - q)) - L1, 1.);
}

} // namespace noa_dcs
