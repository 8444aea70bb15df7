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
 *    lean64 functions (lean64.cuh): same accuracy class, 1 / 2 / 0 / 1 FP64
 *    instructions instead of CUDA's ~30 / 16 / 8 / 8.5, the rest on the
 *    integer and FP32 pipes; divisions by a shared denominator reuse one
 *    reciprocal;
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
using lean64::lean_div;
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

// Clamp of the reference's `if (v < 0.) v = 0.;` that keeps NaN.
__device__ __forceinline__ double clamp0(double v) {
    const long long b = __double_as_longlong(v);
    return (b < 0 && (b & 0x7FFFFFFFFFFFFFFFLL) <= 0x7FF0000000000000LL) ? 0. : v;
}

// Out-of-line copies of the lean64 functions for the two quadrature bodies.
// Inlined, every call site adds ~100 integer and FP32 instructions; the
// photonuclear node (17 transcendental calls) then outgrows the instruction
// cache (ncu: 11.7 "no instruction" stalls per issue) and runs at 87 ms per
// 1e8 pairs against 50 ms with these calls; pair production gains 9%.
// Bremsstrahlung and ionisation, with a few calls each, keep them inlined.
static __device__ __noinline__ double ol_log(double x) { return lean_log(x); }
static __device__ __noinline__ double ol_exp(double x) { return lean_exp(x); }
static __device__ __noinline__ double ol_rcp(double x) { return lean_rcp(x); }
static __device__ __noinline__ double ol_div(double a, double b) { return lean_div(a, b); }

// Whether E (or K) exceeds q by more than a part in 2^10 - 2^11, both of
// ordinary size (2^-62 to 2^97, and q above 2^-94; NaN and negative values
// fail).  There 1 - q / E and K - q keep 42 bits or more whatever the rounding
// of q / E, so that the quotients may be taken lean.  Nearer the edge the
// reference's own rounding shows in the result (by 1 / (1 - q / E) ulp), and
// its IEEE operations are kept.  High words only.
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

// 25 FP64 instructions (42 in the reference's form): the element's factors
// are folded into the two linear forms of each logarithm, Phi_e is taken as
// the logarithm of the inverse, and the scales are one constant.
__device__ __forceinline__ double brems_fp64(double K, double q, const noa_dcs_consts &c) {
    const double E = K + c.mass;
    if (!clear_of_edge(E, q))
        return brems_edge(K, q, c);
    const double invE = lean_rcp(E);
    const double nu = q * invE;
    const double delta = c.br_half_m2 * invE * nu * lean_rcp(1. - nu);
    const double Phi_n = clamp0(lean_log(fma(delta, c.br_n1, c.br_n0) * lean_rcp(fma(delta, c.br_d1, c.br_d0))));
    double Phi_e = 0.;
    if (brems_below(E, q, c))
        Phi_e = clamp0(-lean_log(fma(delta, c.br_e1, c.br_e0) * fma(delta, c.br_f1, ME)));
    const double shape = fma(4. / 3., E * lean_rcp(q), nu - 4. / 3.);
    return clamp0(c.br_scale * fma(c.Zd, Phi_n, Phi_e) * shape);
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
// in s (dcs.hh:188-216), so that it costs one FMA per node:
//   (2 + rho^2)(1 + beta) + xi (3 + rho^2) = a0 + s (a1 - s xf),  xi = xf s
//   5 - rho^2 + 4 beta (1 + rho^2)         = n0 + s n1
//   rho^2 + 2 beta (2 - rho^2)             = -(dc + s ds)
//   (1 + rho^2)(1 + 1.5 beta) - (1 + 2 beta) s / xi = m0 + s m1
//   4 + rho^2 + 3 beta (1 + rho^2)         = q0 + s q1
//   (1 + rho^2)(1.5 + 2 beta)              = e0 + s e1
// c1 = cL / (AZ13 q) scales the screening lengths, which are taken over q.
struct PprodPair {
    double tmin, xf, beta, a0, a1, n0, n1, d1, dc, ds, c1, m0, m1, e0, e1, q0, q1;
};

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
    p.n0 = fma(8., beta, 4.);
    p.n1 = fma(-4., beta, 1.);
    p.d1 = fma(6., beta, 2.);
    p.dc = fma(-2., beta, -1.);
    p.ds = fma(-2., beta, 1.);
    p.c1 = c.pp_2sm * rq;
    p.m0 = fma(p.dc, ol_rcp(p.xf), fma(3., beta, 2.));
    p.m1 = fma(-1.5, beta, -1.);
    p.e0 = fma(4., beta, 3.);
    p.e1 = fma(-2., beta, -1.5);
    p.q0 = fma(6., beta, 5.);
    p.q1 = fma(-3., beta, -1.);
}

// Clamp of the reference's `if (Phi < 0.) Phi = 0.;` for -Phi; keeps NaN.
__device__ __forceinline__ double clamp0_neg(double v) {
    return (unsigned long long)(__double_as_longlong(v) - 1) < 0x7FF0000000000000ULL ? 0. : v;
}

// Node j: w_j (1 - rho) (-2) (Phi_e + Phi_mu / r^2), 51 FP64 instructions (about 75
// in the reference's form) beside 6 logarithms, an exponential and 6
// reciprocals.  The screening logarithms are those of the inverse arguments,
//   Le  = -log(d^2 (1 / xe + cLe)) / 2,   d = 1 / AZ13 + c1 xe / s
//   Lmu = -log(kappa (1 / AZ13 + c1 xmu / s)),
// which spares their products with 1 / d and the square root.
__device__ __forceinline__ double pprod_node(const PprodPair &p, int j, const noa_dcs_consts &c) {
    const double eps = ol_exp(kGL8X[j] * p.tmin);
    const double s = eps * (2. - eps);
    const double xi = p.xf * s;
    const double xi_i = ol_rcp(xi);
    const double opxi = 1. + xi;
    const double inv_opxi = ol_rcp(opxi);
    const double sb = s - p.beta;
    const double crs = p.c1 * ol_rcp(s);

    double Be;
    if (bits_ge(xi, 1E+03))
        Be = xi_i * fma(0.5 * s, p.ds, -p.dc);
    else
        Be = fma(fma(s, fma(-s, p.xf, p.a1), p.a0), ol_log(1. + xi_i), fma(sb, inv_opxi, s - 4.));
    const double Ye = fma(s, p.n1, p.n0) * ol_rcp(fma(p.d1, ol_log(3. + xi_i), fma(s, p.ds, p.dc)));
    const double xe = fma(opxi, Ye, opxi);
    const double de = fma(crs, xe, c.pp_inv_AZ13);
    const double Pe = clamp0_neg(Be * ol_log(de * de * (ol_rcp(xe) + c.pp_cLe)));

    double Bmu;
    if (!bits_ge(xi, 1.0000000000000002E-03))  // xi <= 1e-3
        Bmu = 0.5 * xi * fma(p.beta, 4. - s, 4. + s);
    else
        Bmu = fma(fma(s, p.m1, p.m0), ol_log(opxi), fma(sb, xi * inv_opxi, -p.dc * s));
    const double Ymu = fma(s, p.q1, p.q0) *
                       ol_rcp(fma(fma(s, p.e1, p.e0), ol_log(3. + xi), fma(1.5, s, -0.5)));
    const double xmu = fma(opxi, Ymu, opxi);
    const double Pmu = clamp0_neg(Bmu * ol_log(c.pp_kappa * fma(crs, xmu, c.pp_inv_AZ13)));
    // 1 - rho as the reference rounds it: for small eps its last bit (2^-54 / eps) shows in the result
    return fma(Pmu, c.pp_2_inv_r2, Pe) * (1. - (1. - eps)) * kGL8W[j];
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
    return clamp0(c.pp_cZs * (c.Zd + zeta) * (E - q) * (0.5 * tmin * sum) * ol_rcp(q));
}

// An open pair (pprod_live), its nodes one after the other.
__device__ __forceinline__ double pprod_fp64(double K, double q, const noa_dcs_consts &c) {
    PprodPair p;
    pprod_setup(K, q, c, p);
    double sum = 0.;
#pragma unroll 1  // rolled: smaller code, same FP64 work
    for (int j = 0; j < 8; j++)
        sum += pprod_node(p, j, c);
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

// What one open pair's nodes share.
struct PhotoPair {
    double pc, hd;          // log Q2 = pc + hd x_j
    double h;               // x = h Q2
    double inv_dP, inv_dR;  // 1 / (mP2 + 2 M q), 1 / (mR2 + 2 M q)
    double k2;              // DRSS exponent k1 log Q2 + k2
    double omy, yy, invEE;  // 1 - y, y^2, 1 / E^2
};

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
    p.pc = fma(0.5, log_max, half_min);
    p.hd = fma(0.5, log_max, -half_min);
    p.h = (0.5 / PH_M) * ol_rcp(q);
    p.inv_dP = ol_rcp(fma(2.0 * PH_M, q, 49.457));
    p.inv_dR = ol_rcp(fma(2.0 * PH_M, q, 0.15052));
    p.k2 = fma(c.ph_k1, ol_log(p.h), c.ph_k0);
    const double y = q * invE;
    p.omy = (E - q) * invE;
    p.yy = y * y;
    p.invEE = invE * invE;
}

// Node j: w_j (F2A / (A / 2)) Q2 dds of dcs.hh:289-354, 62 FP64 instructions
// (about 90 in the reference's form) beside 6 logarithms, 10 exponentials and
// 8 reciprocals.  W2 - M2 = Q2 (1/x - 1) = 2 M q - Q2, which makes the
// denominators of xP and xR constants of the pair; log x and log(Q2 / 0.04)
// follow from log Q2 = pc + hd x_j; c1 + (c1 - c2) (1 / (1 + e) - 1) is
// c2 + (c1 - c2) / (1 + e); Q2 / Q2^2 is taken together.
__device__ __forceinline__ double photo_node(const PhotoPair &p, int j, const noa_dcs_consts &c) {
    // ALLM parameters, dcs.hh:262-288.
    const double m02 = 0.31985, mP2 = 49.457, mR2 = 0.15052, Q02 = 0.52544;
    const double cP1 = 0.28067, cP2 = 0.22291, cP3 = 2.1979;
    const double aP1 = -0.0808, aP2 = -0.44812, aP3 = 1.1709;
    const double bP1 = 0.36292, bP2 = 1.8917, bP3 = 1.8439;
    const double cR1 = 0.80107, cR2 = 0.97307, cR3 = 3.4942;
    const double aR1 = 0.58400, aR2 = 0.37888, aR3 = 2.6063;
    const double bR1 = 0.01147, bR2 = 3.7582, bR3 = 0.49338;
    const double inv_lambda2 = 1. / 0.06527;

    const double lq = fma(p.hd, kGL9X[j], p.pc);
    const double Q2 = ol_exp(lq);
    const double invQ2 = ol_rcp(Q2);
    const double x = p.h * Q2;
    // ALLM F2, dcs.hh:289-306
    const double lnt = ol_log(ol_log(ol_log((Q2 + Q02) * inv_lambda2) * c.ph_inv_log_q02));
    const double cP = fma(cP1 - cP2, ol_rcp(1.0 + ol_exp(cP3 * lnt)), cP2);
    const double aP = fma(aP1 - aP2, ol_rcp(1.0 + ol_exp(aP3 * lnt)), aP2);
    const double bP = fma(bP2, ol_exp(bP3 * lnt), bP1);
    const double l1x = ol_log(1. - x);
    double F2 = cP * ol_exp(fma(aP, ol_log((Q2 + mP2) * p.inv_dP), bP * l1x));
    const double cR = fma(cR2, ol_exp(cR3 * lnt), cR1);
    const double aR = fma(aR2, ol_exp(aR3 * lnt), aR1);
    const double bR = fma(bR2, ol_exp(bR3 * lnt), bR1);
    F2 = fma(cR, ol_exp(fma(aR, ol_log((Q2 + mR2) * p.inv_dR), bR * l1x)), F2);
    F2 = Q2 * ol_rcp(Q2 + m02) * F2;
    // DRSS shadowing, dcs.hh:310-319
    if (!bits_ge(x, 0.0014))
        F2 *= c.ph_a_low;
    else if (!bits_ge(x, 0.04))
        F2 *= ol_exp(fma(c.ph_k1, lq, p.k2));
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
    const double t = fma(-c.ph_m2, invQ2, 0.5) * fma(Q2, p.invEE, p.yy);
    const double dds = fma(fma(t, ol_rcp(R1), p.omy), invQ2, -0.25 * p.invEE);
    return F2 * dds * kGL9W[j];
}

__device__ __forceinline__ double photo_finish(double K, double q, double hd, double sum, const noa_dcs_consts &c) {
    return clamp0(c.ph_scale_A * sum * hd * (K + c.mass) * ol_rcp(q));
}

// An open pair (photo_live), its nodes one after the other.
__device__ __forceinline__ double photo_fp64(double K, double q, const noa_dcs_consts &c) {
    PhotoPair p;
    photo_setup(K, q, c, p);
    double sum = 0.;
#pragma unroll 1
    for (int j = 0; j < 9; j++)
        sum += photo_node(p, j, c);
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
