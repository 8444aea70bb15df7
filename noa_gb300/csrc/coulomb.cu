/*
 * Elastic (Coulomb) scattering per kinetic energy, FP64:
 *
 *   coulomb_data       dcs.hh:499-622  CM Lorentz factors, spin factor,
 *                                      screening parameters + pole factors,
 *                                      inverse Wentzel path
 *   coulomb_transport  dcs.hh:624-699  first two transport coefficients
 *                                      below a cut-off angle mu
 *   hard_scattering    dcs.hh:702-872  hard-scattering cut-off angle mu0 and
 *                                      mean free path lb_h over nel elements,
 *                                      by Ridders' method (numerics.hh:154-216)
 *
 * This translation unit is compiled with -fmad=false so that every product
 * and sum is rounded as in the reference (no FMA contraction); the Ridders
 * iteration branches on the signs of objective values, and a contracted
 * expression could change its path.  pow(A, 1/3), pow(Z, 2/3) and the
 * maximum hard angle are per-element constants computed once on the host
 * with the C library (the reference computes the same values per call).
 *
 * These are scalar, branchy, per-K computations (a few logs, a series of
 * 10 + Z terms, up to 100 root iterations), bound by the FP64 pipe when there
 * are enough energies and by latency when there are not: CTAs of one warp
 * spread the energies over the SMs, divisions take 3 FP64 instructions
 * (lean64::qdiv), the transport coefficients give a pole a lane where energies are
 * few, and the hard-scattering search an energy up to 32 (hard_scattering_kernel).  Records are the
 * reference's: fCM [n][2], screen [n][9].
 */
#include "dcs_launch.h"
#include "lean64.cuh"

#include <cuda_runtime.h>

namespace noa_coulomb {

constexpr int NSF = 9;
constexpr int C_THREADS = 32;
constexpr double ATOMIC_MASS_ENERGY = 0.931494;  // physics.hh:55
constexpr double KIN_CUTOFF = 1E-9;              // physics.hh:78
constexpr double EHS_PATH_MAX = 1E+9;            // physics.hh:79
constexpr double EHS_OVER_MSC = 1E-4;            // physics.hh:80

using lean64::qdiv;
using lean64::qdiv_fast;

// std::min's rule (b < a ? b : a), which differs from fmin for NaN.
__device__ __forceinline__ double smin(double a, double b) { return (b < a) ? b : a; }

__device__ __forceinline__ double frame_parameters(double *fCM, double K, const noa_coulomb_element &e, double mass) {
    const double Ma = e.A * ATOMIC_MASS_ENERGY;
    double M2 = mass + Ma;
    M2 *= M2;
    const double sCM12i = qdiv(1., sqrt(M2 + 2. * Ma * K));
    fCM[0] = (K + mass + Ma) * sCM12i;
    double kinetic0 = (K * Ma + mass * (mass + Ma)) * sCM12i - mass;
    if (kinetic0 < KIN_CUTOFF)
        kinetic0 = KIN_CUTOFF;
    const double etot = K + mass + Ma;
    const double betaCM2 = qdiv(K * (K + 2. * mass), etot * etot);
    double rM2 = qdiv(mass, Ma);
    rM2 *= rM2;
    fCM[1] = sqrt(rM2 * (1. - betaCM2) + betaCM2);
    return kinetic0;
}

__device__ __forceinline__ double screening_parameters(double *ps, double K, const noa_coulomb_element &e,
                                                       double mass) {
    const double R1 = 1.02934 * e.A13 + 0.435;
    const double R2 = 2.;
    const double p2 = K * (K + 2. * mass);
    const double d = qdiv(5.8406E-02, p2);
    ps[1] = qdiv(d, R1 * R1);
    ps[2] = qdiv(d, R2 * R2);

    // Moliere atomic screening with Kuraev's Coulomb correction, dcs.hh:560-590
    const int Z = e.Z;
    const double etot = K + mass;
    const double ZE = Z * etot;
    const double zeta2 = qdiv(5.3251346E-05 * (ZE * ZE), p2);
    double cK;
    if (zeta2 > 1.) {
        // the reference's sum in its order; the quotients of four terms do not
        // wait for one another (1 < zeta2 < 2^100 keeps them in qdiv's range)
        const int n = 10 + Z;
        const bool fast = zeta2 < 0x1p100;
        double f = 0.;
        for (int i = 1; i <= n; i += 4) {
            double term[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const double id = (double)(i + k);
                const double den = id * ((double)((i + k) * (i + k)) + zeta2);
                term[k] = fast ? qdiv_fast(zeta2, den) : zeta2 / den;
            }
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (i + k <= n)
                    f += term[k];
        }
        cK = exp(f);
    } else {
        cK = exp(1. - qdiv(1., 1. + zeta2) + zeta2 * (0.2021 + zeta2 * (0.0083 * zeta2 - 0.0369)));
    }
    const double cM = 1. + 3.34 * zeta2;
    double r = qdiv(K, etot);
    r *= r;
    const double c = r * cK + (1. - r) * cM;
    ps[0] = qdiv(5.179587126E-12 * e.Z23 * c, p2);

    // pole reduction factors, dcs.hh:592-599
    const double d01 = qdiv(1., ps[0] - ps[1]);
    const double d02 = qdiv(1., ps[0] - ps[2]);
    const double d12 = qdiv(1., ps[1] - ps[2]);
    ps[6] = d01 * d01 * d02 * d02;
    ps[7] = d01 * d01 * d12 * d12;
    ps[8] = d12 * d12 * d02 * d02;
    ps[3] = 2. * ps[6] * (d01 + d02);
    ps[4] = 2. * ps[7] * (d12 - d01);
    ps[5] = -2. * ps[8] * (d12 + d02);

    // inverse Wentzel path, dcs.hh:531-538
    const double dw = qdiv(K * (K + 2. * mass), Z * (K + mass));
    return qdiv(1., e.A * 2.54910918E+08 * ps[0] * (1. + ps[0]) * dw * dw);
}

__global__ void __launch_bounds__(C_THREADS) coulomb_data_kernel(const double *__restrict__ K, int64_t n,
                                                           const noa_coulomb_element e, double mass,
                                                           double *__restrict__ fCM, double *__restrict__ screen,
                                                           double *__restrict__ fspin,
                                                           double *__restrict__ invlambda) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double f[2], ps[NSF];
        const double kinetic0 = frame_parameters(f, K[i], e, mass);
        const double ek = kinetic0 + mass;  // spin factor, dcs.hh:525-528
        fspin[i] = qdiv(kinetic0 * (ek + mass), ek * ek);
        invlambda[i] = screening_parameters(ps, kinetic0, e, mass);
        fCM[2 * i] = f[0];
        fCM[2 * i + 1] = f[1];
#pragma unroll
        for (int j = 0; j < NSF; j++)
            screen[NSF * i + j] = ps[j];
    }
}

// Pole i's share of the coefficients, dcs.hh:639-672: s = screen[i], a and b its
// factors.
__device__ __forceinline__ void transport_term(double s, double a, double b, double fspin, double mu, double mu2,
                                               double &t0, double &t1) {
    double r = qdiv(mu, mu + s);
    double L = log(1. + qdiv(mu, s));
    double mu1 = mu;
    const double I0 = qdiv(r, s);
    const double J0 = L;
    const double I1 = L - r;
    r *= s;
    L *= s;
    const double J1 = mu1 - L;
    const double I2 = mu1 - 2. * L + r;
    L *= s;
    mu1 *= s;
    const double J2 = mu2 + L - mu1;
    t0 = a * (J0 - fspin * J1) + b * (I0 - fspin * I1);
    t1 = a * (J1 - fspin * J2) + b * (I1 - fspin * I2);
}

// dcs.hh:624-677, an energy by W lanes (1: all poles in one thread, 4: a lane a
// pole, added in the reference's order by shuffles).
template <int W>
__global__ void __launch_bounds__(C_THREADS) coulomb_transport_kernel(const double *__restrict__ screen,
                                                                const double *__restrict__ fspin,
                                                                const double *__restrict__ mu_, int64_t n_mu,
                                                                int64_t n, double *__restrict__ coefs) {
    constexpr int PER = C_THREADS / W;
    const int lane = threadIdx.x % W, first = threadIdx.x - lane, pole = lane < 3 ? lane : 2;
    for (int64_t base = blockIdx.x * (int64_t)PER; base < n; base += (int64_t)gridDim.x * PER) {  // warp-uniform
        const int64_t at = base + threadIdx.x / W, i = at < n ? at : n - 1;
        const double *s = screen + NSF * i;
        const double s0 = s[0], s1 = s[1], s2 = s[2], spin = fspin[i], mu = mu_[n_mu == 1 ? 0 : i];
        const double nuclear_screening = (s1 < s2) ? s1 : s2;
        const bool tiny = mu < 1E-08 * nuclear_screening;
        double out0 = 0., out1 = 0.;
        // with W > 1 decided for the warp: its lanes exchange terms
        if (W == 1 ? !tiny : __any_sync(0xFFFFFFFFu, !tiny)) {
            const double mu2 = 0.5 * mu * mu;
            double t0[3], t1[3];
            if constexpr (W == 1) {
#pragma unroll
                for (int j = 0; j < 3; j++)
                    transport_term(s[j], s[3 + j], s[6 + j], spin, mu, mu2, t0[j], t1[j]);
            } else {
                double a, b;
                transport_term(s[pole], s[3 + pole], s[6 + pole], spin, mu, mu2, a, b);
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    t0[j] = __shfl_sync(0xFFFFFFFFu, a, first + j);
                    t1[j] = __shfl_sync(0xFFFFFFFFu, b, first + j);
                }
            }
            double c0 = 0., c1 = 0.;
#pragma unroll
            for (int j = 0; j < 3; j++) {
                c0 += t0[j];
                c1 += t1[j];
            }
            const double kk = s0 * (1. + s0) * s1 * s1 * s2 * s2;
            out0 = c0 * kk;
            out1 = c1 * (2. * kk);
        }
        if (tiny) {
            const double L = log(1. + qdiv(mu, s0));
            const double r = qdiv(mu, mu + s0);
            const double k = s0 * (1. + s0);
            out0 = k * (qdiv(r, s0) - spin * (L - r));
            const double I2 = mu - s0 * (r - 2. * L);
            out1 = 2. * k * (L - r - spin * I2);
        }
        if (at < n && lane == 0) {
            coefs[2 * i] = out0;
            coefs[2 * i + 1] = out1;
        }
    }
}

struct HardArgs {
    const double *G, *fCM, *screen, *invlambda, *fspin;
    int64_t nel, nkin;
};

// W lanes that share one energy: the lanes of a warp in groups of W.
template <int W>
struct Group {
    unsigned mask;
    int lane, first;  // within the group, and the group's first lane
    __device__ __forceinline__ Group() {
        const int l = threadIdx.x & 31;
        lane = l % W;
        first = l - lane;
        mask = W == 32 ? 0xFFFFFFFFu : ((1u << W) - 1u) << first;
    }
    __device__ __forceinline__ double from(double v, int l) const {
        return W == 1 ? v : __shfl_sync(mask, v, first + l);
    }
};

// Term i of the restricted cross-section of one element (dcs.hh:702-740),
// with what the element's other terms and its asymptotic form need.
struct Term {
    double s, a, b;  // screen[i], screen[3 + i], screen[6 + i]
    double s0, kfac, nuclear, fspin, inv;
};

__device__ __forceinline__ void load_term(Term &t, const HardArgs &h, int64_t iel, int64_t i, int term) {
    const int64_t off = iel * h.nkin + i;
    const double *s = h.screen + NSF * off;
    const double s0 = s[0], s1 = s[1], s2 = s[2];
    t.s = s[term];
    t.a = s[3 + term];
    t.b = s[6 + term];
    t.s0 = s0;
    t.kfac = s0 * (1. + s0) * s1 * s1 * s2 * s2;
    t.nuclear = (s1 < s2) ? s1 : s2;
    t.fspin = h.fspin[off];
    t.inv = h.invlambda[off];
}

__device__ __forceinline__ double eval_term(const Term &t, double mu, bool asymptotic) {
    const double sm = t.s + mu, sp = t.s + 1.;
    // lean_log rounds as correctly as glibc's log here (0.1 - 0.2% of its last
    // bits differ from the exact value's, 0.13% of glibc's), which the root
    // search needs: of 40000 energies x 10 elements 1.0% of mu0 and 1.1% of
    // lb_h differ from the reference's in any bit, as with CUDA's log, at half
    // its time (n = 20000: 2.32 ms with CUDA's log, 1.4 ms).
    const double L = lean64::lean_log(qdiv(sp, sm));
    const double r = qdiv(1. - mu, sm * sp);
    if (asymptotic)
        return r - t.fspin * (L - t.s * r);
    const double I0 = r, J0 = L, I1 = L - t.s * r, J1 = mu - t.s * L;
    return t.a * (J0 - t.fspin * J1) + t.b * (I0 - t.fspin * I1);
}

// dcs.hh:742-752 for energy index i: element-summed restricted cross-section
// less cs_h, in every lane of the group.  E = W / 3 elements at a time, a
// lane a (element, term); the terms of an element and the elements are added
// in the reference's order.  W = 1: one lane, term by term.
template <int W>
__device__ __forceinline__ double objective(const Group<W> &g, const HardArgs &h, int64_t i, const Term &mine,
                                            double cs_h, double mu) {
    double cs_tot = 0.;
    const bool none = mu >= 1.;  // the restricted cross-section is 0
    if constexpr (W == 1) {
        for (int64_t iel = 0; iel < h.nel; iel++) {
            Term t;
            load_term(t, h, iel, i, 0);
            const bool asymptotic = mu < 1E-08 * t.nuclear;
            double cs = none ? 0. : eval_term(t, mu, asymptotic);
            if (asymptotic) {
                cs = t.s0 * (1. + t.s0) * cs;
            } else if (!none) {
#pragma unroll 1
                for (int k = 1; k < 3; k++) {
                    load_term(t, h, iel, i, k);
                    cs += eval_term(t, mu, false);
                }
                cs = t.kfac * cs;
            }
            cs_tot += t.inv * cs;
        }
    } else {
        constexpr int E = W / 3;
        const int el = g.lane / 3;
        for (int64_t e0 = 0; e0 < h.nel; e0 += E) {
            const bool valid = el < E && e0 + el < h.nel;
            Term t = mine;  // the first E elements' terms stay in registers
            if (e0 > 0 && valid)
                load_term(t, h, e0 + el, i, g.lane % 3);
            double v = 0.;
            const bool asymptotic = mu < 1E-08 * t.nuclear;
            if (valid && !none)
                v = eval_term(t, mu, asymptotic);
            const int b = el < E ? 3 * el : 0;
            const double v0 = g.from(v, b), v1 = g.from(v, b + 1), v2 = g.from(v, b + 2);
            const double cs = none ? 0. : (asymptotic ? t.s0 * (1. + t.s0) * v0 : t.kfac * ((v0 + v1) + v2));
            const double w = t.inv * cs;
            const int m = h.nel - e0 < E ? (int)(h.nel - e0) : E;
            for (int e = 0; e < m; e++)
                cs_tot += g.from(w, 3 * e);
        }
    }
    return cs_tot - cs_h;
}

// Ridders' method, numerics.hh:154-216; false where the reference returns
// an empty optional.
template <int W>
__device__ __forceinline__ bool ridders(const Group<W> &g, const HardArgs &a, int64_t i, const Term &mine, double cs_h,
                                        double xa, double xb, double fa, double fb, double xtol, double rtol,
                                        int max_iter, double &root) {
    if (fa * fb > 0)
        return false;
    if (fa == 0) {
        root = xa;
        return true;
    }
    if (fb == 0) {
        root = xb;
        return true;
    }
    const double tol = xtol + rtol * smin(fabs(xa), fabs(xb));
#pragma unroll 1
    for (int it = 0; it < max_iter; it++) {
        double dm = 0.5 * (xb - xa);
        const double xm = xa + dm;
        double x = xm, fm = 0., fn = 0.;
#pragma unroll 1
        for (int half = 0; half < 2; half++) {  // one copy of the objective
            const double f = objective<W>(g, a, i, mine, cs_h, x);
            if (half == 0) {
                fm = f;
                double sgn = (fb > fa) ? 1. : -1.;
                double dn = qdiv(sgn * dm * fm, sqrt(fm * fm - fa * fb));
                sgn = (dn > 0.) ? 1. : -1.;
                dn = fabs(dn);
                dm = fabs(dm) - 0.5 * tol;
                if (dn < dm)
                    dm = dn;
                x = xm - sgn * dm;
            } else {
                fn = f;
            }
        }
        const double xn = x;
        if (fn * fm < 0.0) {
            xa = xn;
            fa = fn;
            xb = xm;
            fb = fm;
        } else if (fn * fa < 0.0) {
            xb = xn;
            fb = fn;
        } else {
            xa = xn;
            fa = fn;
        }
        if (fn == 0.0 || fabs(xb - xa) < tol) {
            root = xn;
            return true;
        }
    }
    return false;
}

// W lanes an energy.  An energy's search is a chain of 20 - 40 objectives of
// nel x 3 terms (a logarithm and two divisions each): one lane an energy took
// 1.9 ms for 5003 energies x 10 elements, on 40 SMs; with a lane a term the
// objectives take one term's time and the energies reach every SM (0.4 ms,
// bound by the FP64 pipe).  The
// redundant rest of the search costs the group nothing (all lanes of a warp
// issue together).
template <int W>
__global__ void __launch_bounds__(C_THREADS) hard_scattering_kernel(const HardArgs a, double max_mu0,
                                                                    double *__restrict__ mu0_out,
                                                                    double *__restrict__ lb_h_out) {
    const Group<W> g;
    constexpr int per_cta = C_THREADS / W;
    for (int64_t i = blockIdx.x * (int64_t)per_cta + threadIdx.x / W; i < a.nkin; i += (int64_t)gridDim.x * per_cta) {
        Term mine = {};
        if (W > 1 && g.lane < 3 * (W / 3) && g.lane / 3 < a.nel)
            load_term(mine, a, g.lane / 3, i, g.lane % 3);
        // sums over the elements, a lane an element, added in element order
        double invlb_m = 0., invlb1_m = 0., s_m_l = 0., s_m_h = 0.;
        for (int64_t e0 = 0; e0 < a.nel; e0 += W) {
            double m = 0., h = 0., l = 0., m1 = 0.;
            if (e0 + g.lane < a.nel) {
                const int64_t off = (e0 + g.lane) * a.nkin + i;
                const double invlb = a.invlambda[off];
                const double scr = a.screen[NSF * off];
                m = invlb * a.G[2 * off];
                h = scr * invlb;
                l = qdiv(invlb, scr);
                const double d = qdiv(1., a.fCM[2 * off] * (1. + a.fCM[1 + 2 * off]));
                m1 = invlb * a.G[1 + 2 * off] * d * d;
            }
            const int n = a.nel - e0 < W ? (int)(a.nel - e0) : W;
            for (int e = 0; e < n; e++) {
                invlb_m += g.from(m, e);
                s_m_h += g.from(h, e);
                s_m_l += g.from(l, e);
                invlb1_m += g.from(m1, e);
            }
        }
        const double lb_m = qdiv(1., invlb_m);
        double lb_h = smin(qdiv(EHS_OVER_MSC, invlb1_m), EHS_PATH_MAX);
        double mu0;
        if (!(lb_m < lb_h)) {
            lb_h = lb_m;
            mu0 = 0;
        } else {
            const double s_m = (lb_h > 2. * lb_m) ? s_m_h * lb_m : qdiv(1., s_m_l * lb_m);
            mu0 = qdiv(s_m * (lb_h - lb_m), s_m * lb_h + lb_m);
            const double cs_h = qdiv(1., lb_h);
            double mu_max = smin(4. * mu0, 1.);
            double mu_min = 0.25 * mu0;
            double fmax = objective<W>(g, a, i, mine, cs_h, mu_max);
            // fmax > 0: the reference keeps the asymptotic mu0 and lb_h
            if (!(fmax > 0.)) {
                double fmin_ = objective<W>(g, a, i, mine, cs_h, mu_min);
                if (fmin_ < 0.) {
                    mu_max = mu_min;
                    fmax = fmin_;
                    mu_min = 0.;
                    fmin_ = objective<W>(g, a, i, mine, cs_h, mu_min);
                }
                if (mu_min < max_mu0) {
                    mu_max = smin(mu_max, max_mu0);
                    double root;
                    if (ridders<W>(g, a, i, mine, cs_h, mu_min, mu_max, fmin_, fmax, 1E-6 * mu0, 1E-6, 100, root))
                        mu0 = root;
                }
                mu0 = smin(mu0, max_mu0);
                lb_h = objective<W>(g, a, i, mine, cs_h, mu0) + cs_h;
                lb_h = (lb_h <= 1. / EHS_PATH_MAX) ? EHS_PATH_MAX : qdiv(1., lb_h);
            }
        }
        if (g.lane == 0) {
            mu0_out[i] = mu0;
            lb_h_out[i] = lb_h;
        }
    }
}

int sm_count() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

int grid_for(int64_t n, int per_cta, int sms) {
    const int64_t blocks = (n + per_cta - 1) / per_cta;
    const int64_t cap = (int64_t)sms * 1024;
    return (int)(blocks < cap ? blocks : cap);
}

} // namespace noa_coulomb

using namespace noa_coulomb;

cudaError_t noa_dcs_launch_coulomb_data(const double *K, int64_t n, const noa_coulomb_element *e, double mass,
                                        double *fCM, double *screen, double *fspin, double *invlambda,
                                        cudaStream_t stream) {
    if (n <= 0)
        return cudaSuccess;
    coulomb_data_kernel<<<grid_for(n, C_THREADS, sm_count()), C_THREADS, 0, stream>>>(K, n, *e, mass, fCM, screen,
                                                                                      fspin, invlambda);
    return cudaGetLastError();
}

// Energies per SM up to which a pole has a lane of its own: one warp of whole
// energies an SM waits 9.8 us for 1660 dependent instructions, four lanes an
// energy 4.5 us up to one warp (1000 energies 4.7 against 9.8, 5003 energies 6.1
// against 9.8), while with more the FP64 pipe fills and the idle fourth lane
// costs (12000 energies 9.6 / 9.9, 20000 15.8 / 12.8, 1e5 67 / 45).
constexpr int64_t TRANSPORT_LANES = 64;

cudaError_t noa_dcs_launch_coulomb_transport(const double *screen, const double *fspin, const double *mu,
                                             int64_t n_mu, int64_t n, double *coefs, cudaStream_t stream) {
    if (n <= 0)
        return cudaSuccess;
    const int sms = sm_count();
    if (n <= TRANSPORT_LANES * (int64_t)sms)
        coulomb_transport_kernel<4><<<grid_for(n, C_THREADS / 4, sms), C_THREADS, 0, stream>>>(screen, fspin, mu, n_mu,
                                                                                              n, coefs);
    else
        coulomb_transport_kernel<1><<<grid_for(n, C_THREADS, sms), C_THREADS, 0, stream>>>(screen, fspin, mu, n_mu, n,
                                                                                          coefs);
    return cudaGetLastError();
}

namespace {

template <int W>
cudaError_t launch_hard(const HardArgs &a, double max_mu0, double *mu0, double *lb_h, int sms, cudaStream_t stream) {
    hard_scattering_kernel<W><<<grid_for(a.nkin, C_THREADS / W, sms), C_THREADS, 0, stream>>>(a, max_mu0, mu0, lb_h);
    return cudaGetLastError();
}

} // namespace

cudaError_t noa_dcs_launch_hard_scattering(const double *G, const double *fCM, const double *screen,
                                           const double *invlambda, const double *fspin, int64_t nel, int64_t nkin,
                                           double max_mu0, double *mu0, double *lb_h, cudaStream_t stream) {
    if (nkin <= 0)
        return cudaSuccess;
    HardArgs a{G, fCM, screen, invlambda, fspin, nel, nkin};
    const int sms = sm_count();
    // As many lanes an energy as there are terms, while that many threads fit
    // the chip about twice (1024 an SM); then fewer, down to one lane an energy,
    // which wastes no lane (3 of 4 work with one element and W = 4, 30 of 32
    // with ten and W = 32).
    const int64_t room = (int64_t)sms * 1024;
    if (nel > 5 && nkin * 32 <= 2 * room)
        return launch_hard<32>(a, max_mu0, mu0, lb_h, sms, stream);
    if (nel > 2 && nkin * 16 <= 2 * room)
        return launch_hard<16>(a, max_mu0, mu0, lb_h, sms, stream);
    if (nel > 1 && nkin * 8 <= 2 * room)
        return launch_hard<8>(a, max_mu0, mu0, lb_h, sms, stream);
    if (nkin * 4 <= 2 * room)
        return launch_hard<4>(a, max_mu0, mu0, lb_h, sms, stream);
    return launch_hard<1>(a, max_mu0, mu0, lb_h, sms, stream);
}
