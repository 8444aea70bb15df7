/*
 * Recoil-energy integrals of the DCS per kinetic energy (FP64):
 *
 *   DEL: (1/E) int_{K xlow}^{K} q dsigma/dq dq      (moment 0)
 *   CEL: (1/E) int_{K xlow}^{K} q^2 dsigma/dq dq    (moment 1)
 *
 * Reference: recoil_integral (src/noa/pms/dcs.hh:89-105) with del_integrand /
 * cel_integrand (:107-113), mapped by vmap_integral (:115-130): a composite
 * 6-node Gauss-Legendre rule (numerics.hh:71-108) over t = log q with
 * n_itv = ceil(min_points / 6) intervals, i.e. 6 n_itv DCS evaluations per
 * K; ionisation switches to its closed form below the radiative-correction
 * threshold (dcs.hh:446-496, 955-1001).
 *
 * Kernel: a CTA takes a tile of kpt kinetic energies and all their nodes
 * (kpt * nodes pairs, at most 1536).  Each pair (K, q_i) is classified with the
 * process's exact bounds; closed pairs contribute 0, open ones go to the
 * shared-memory work queue and are evaluated in batches with every lane busy,
 * the two quadrature processes a (pair, node) a thread (quad_batch).  Each
 * weighted node value lands in a shared array indexed by (K, node), and one
 * warp per K then sums its nodes in a fixed order, so the result does not
 * depend on scheduling.
 *
 * kpt and the CTA's width follow the number of energies (integral_width): a
 * table of 146 energies has one energy a CTA and up to 1024 threads on it (a
 * 9-node photonuclear batch of 8 energies in 256 threads kept 19 of 152 SMs
 * busy for 740 us); a fine grid has 8 energies a CTA of 128 threads, five or
 * six CTAs an SM.
 */
#include "dcs_quad.cuh"

#include <cuda_runtime.h>

namespace noa_dcs {

constexpr int I_PAIRS = 1536;  // pairs per tile (kpt * nodes <= I_PAIRS)
constexpr int I_KMAX = 128;    // kinetic energies per tile at most

// CTA widths: many energies / at most two per SM / at most one.
constexpr int I_NARROW = 128, I_MID = 256, I_WIDE = 1024;
// Pairs per batch of the quadrature processes -- all nodes of an energy in the
// wider CTAs (180 and 300 nodes are usual), as each batch waits once for its
// pairs' setup and once for their end -- and the resident CTAs that the
// kernels are compiled for.
constexpr int i_batch(int threads) { return threads == I_WIDE ? 320 : (threads == I_MID ? 192 : 128); }
constexpr int i_ctas(int threads) { return threads == I_WIDE ? 1 : (threads == I_MID ? 2 : 5); }
// A queue drained below `batch` after every step holds up to batch - 1 entries
// when the next step's `threads` arrive.
constexpr int queue_capacity(int batch, int threads) { return batch - 1 + threads; }

__constant__ double kGL6X[6] = {0.03376524, 0.16939531, 0.38069041, 0.61930959, 0.83060469, 0.96623476};
__constant__ double kGL6W[6] = {0.08566225, 0.18038079, 0.23395697, 0.23395697, 0.18038079, 0.08566225};

struct IntegralParams {
    const double *K;
    double *out;
    int64_t n;
    double xlow;
    int nodes;  // 6 * n_itv
    int n_itv;
    int kpt;    // kinetic energies per tile
    int moment; // 0 = DEL, 1 = CEL
};

template <int PROC>
__device__ __forceinline__ bool i_open(double K, double q, const noa_dcs_consts &c) {
    if (PROC == NOA_DCS_PROC_PPROD)
        return pprod_live(K, q, c);
    else if (PROC == NOA_DCS_PROC_PHOTO)
        return photo_live(K, q, c);
    else if (PROC == NOA_DCS_PROC_ION) {
        // ionisation's early returns, dcs.hh:415-424
        const int first = ion_first_exit(K, q, c);
        if (first >= 0)
            return first && !bits_ge(c.io_Wmin, q);
        const double P2 = K * (K + 2. * c.mass);
        const double Wmax = ion_wmax(P2, K + c.mass, c);
        return !((Wmax < NOA_X_FRACTION * K) || (q > Wmax) || (q <= c.io_Wmin));
    } else
        return true;
}

// The closed-form ionisation integrals, dcs.hh:446-496 (FP64, IEEE order).
__device__ __forceinline__ double ion_analytic(double K, double xlow, int moment, const noa_dcs_consts &c) {
    const double mass = c.mass;
    const double P2 = K * (K + 2. * mass);
    const double E = K + mass;
    const double Wmax = ion_wmax(P2, E, c);
    if (Wmax < NOA_X_FRACTION * K)
        return 0.;
    double Wmin = c.io_Wmin;
    const double qlow = K * xlow;
    if (qlow >= Wmin)
        Wmin = qlow;
    if (Wmax <= Wmin)
        return 0.;
    const double a0 = x_div(0.5, P2), a1 = x_div(-1., Wmax), a2 = x_div(E * E, P2);
    const double lw = log(x_div(Wmax, Wmin));
    double term;
    if (moment == 0)
        term = x_add(x_add(x_mul(a0, Wmax - Wmin), x_mul(a1, lw)), x_mul(a2, x_sub(x_div(1., Wmin), x_div(1., Wmax))));
    else
        term = x_add(x_add(x_mul(x_mul(0.5, a0), x_sub(x_mul(Wmax, Wmax), x_mul(Wmin, Wmin))), x_mul(a1, Wmax - Wmin)),
                     x_mul(a2, lw));
    return x_mul(x_div(x_mul(1.535336E-05, c.Zd), c.A), term);
}

// Weighted value of a node, f h w of numerics.hh:86, from its DCS d (f = d q
// or d q^2).
__device__ __forceinline__ double i_weighted(double d, double q, double h, int node, int moment) {
    const double f = moment == 0 ? x_mul(d, q) : x_mul(x_mul(d, q), q);
    return x_mul(x_mul(f, h), kGL6W[node % 6]);
}

// The sum of a kinetic energy's node values by one warp, in every lane: lane
// sums of every 32nd node, then a butterfly -- one fixed order, whatever the
// scheduling.  (One thread's node-ordered sum of 180 nodes was 180 dependent
// additions, 6 us at the end of a tile.)
__device__ __forceinline__ double warp_node_sum(const double *v, int nodes) {
    double s = 0.;
    for (int i = threadIdx.x & 31; i < nodes; i += 32)
        s += v[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

template <int PROC, int THREADS>
__global__ void __launch_bounds__(THREADS, i_ctas(THREADS))
    recoil_integral_kernel(const IntegralParams p, const noa_dcs_consts c) {
    extern __shared__ double vals[];  // weighted node values of the tile, [k][node]
    constexpr int I_BATCH = i_batch(THREADS);
    constexpr int batch = is_quad(PROC) ? I_BATCH : THREADS;
    constexpr int QCAP = queue_capacity(batch, THREADS);
    __shared__ double qQ[QCAP];  // queued recoil energies
    __shared__ int qS[QCAP];     // their slots in vals
    __shared__ QuadSmem<PROC, I_BATCH> quad;
    __shared__ double sK[I_KMAX], sLb[I_KMAX], sH[I_KMAX];
    __shared__ int warp_tot[THREADS / 32];
    __shared__ int tile_open;
    const int pairs = p.kpt * p.nodes;
    const int64_t tiles = (p.n + p.kpt - 1) / p.kpt;
    const double ion_thr = c.io_k_rad;  // 0.5 (m - me)^2 / me, dcs.hh:962-963

    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t k0 = tile * p.kpt;
        if ((int)threadIdx.x < p.kpt) {
            // bounds of the t = log q rule for this K, numerics.hh:80-81
            const int64_t ki = k0 + threadIdx.x;
            const double K = ki < p.n ? p.K[ki] : 1.;
            const double lb = log(K * p.xlow), ub = log(K);
            sK[threadIdx.x] = K;
            sLb[threadIdx.x] = lb;
            sH[threadIdx.x] = x_div(ub - lb, fpconv::f64i(p.n_itv));
        }
        __syncthreads();
        int qn = 0;
        for (int base = 0;; base += THREADS) {
            const bool more = base < pairs;  // block-uniform
            if (more) {
                const int slot = base + threadIdx.x;
                bool open = false;
                double q = 0.;
                if (slot < pairs) {
                    const int kk = slot / p.nodes, i = slot - kk * p.nodes;
                    vals[slot] = 0.;
                    const double K = sK[kk];
                    if (k0 + kk < p.n && !(PROC == NOA_DCS_PROC_ION && K <= ion_thr)) {
                        // node i of the composite rule, numerics.hh:84-86, in IEEE order
                        const double t = x_add(sLb[kk], x_mul(sH[kk], fpconv::f64i(i / 6) + kGL6X[i % 6]));
                        q = lean_exp(t);
                        open = i_open<PROC>(K, q, c);
                    }
                }
                const int pos = qn + block_scan<THREADS>(open ? 1 : 0, warp_tot, &tile_open);
                if (open) {
                    qQ[pos] = q;
                    qS[pos] = slot;
                }
                __syncthreads();
                qn += tile_open;
            }
            // one call site of the evaluation (a pair's rounding must not
            // depend on its queue position): full batches, then the rest
            while (qn >= batch || (!more && qn > 0)) {
                const int take = qn < batch ? qn : batch;
                const int first = qn - take;
                if constexpr (is_quad(PROC)) {
                    quad_batch<PROC, THREADS>(
                        quad, take, c,
                        [&](int e, double &K, double &q) {
                            K = sK[qS[first + e] / p.nodes];
                            q = qQ[first + e];
                        },
                        [&](int e, double d) {
                            const int sl = qS[first + e], kk = sl / p.nodes;
                            vals[sl] = i_weighted(d, qQ[first + e], sH[kk], sl - kk * p.nodes, p.moment);
                        });
                } else if ((int)threadIdx.x < take) {
                    const int sl = qS[first + threadIdx.x], kk = sl / p.nodes;
                    const double K = sK[kk], q = qQ[first + threadIdx.x];
                    const double d = PROC == NOA_DCS_PROC_BREMS ? brems_fp64(K, q, c) : ion_fp64(K, q, c);
                    vals[sl] = i_weighted(d, q, sH[kk], sl - kk * p.nodes, p.moment);
                }
                qn -= take;
                __syncthreads();
            }
            if (!more)
                break;
        }
        // one warp per kinetic energy
        for (int kk = threadIdx.x >> 5; kk < p.kpt && k0 + kk < p.n; kk += THREADS / 32) {
            const double s = warp_node_sum(vals + kk * p.nodes, p.nodes);
            if ((threadIdx.x & 31) == 0) {
                const double K = sK[kk];
                p.out[k0 + kk] = (PROC == NOA_DCS_PROC_ION && K <= ion_thr) ? ion_analytic(K, p.xlow, p.moment, c)
                                                                            : x_div(s, K + c.mass);
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------ soft-scattering transport
/*
 * soft_scattering (dcs.hh:941-952) per K: the closed-form ionisation part
 * (dcs.hh:874-899) plus twice a 6-node composite GL rule over
 * t = log(nu / X_FRACTION) on [log 1e-6, 0] with 17 intervals (102 nodes) of
 * photonuclear(K, q) * ratio(K, q) * nu, q = nu K, where ratio is the
 * mu-integrated angular weight of dcs.hh:911-934.  Same tile / queue scheme
 * as the recoil integrals: closed photonuclear nodes contribute
 * 0 * ratio * nu (0, or NaN where the weight is not finite, as in the
 * reference), open ones are evaluated in batches of 128 or 192.
 */
constexpr int S_NODES = 102;             // 6 * ceil(100 / 6)
constexpr int S_KMAX = 8;                // kinetic energies per tile at most

struct SoftParams {
    const double *K;
    double *out;
    int64_t n;
    double lb;  // log(1e-6)
    double h;   // -lb / 17
    int kpt;    // kinetic energies per tile
};

// The mu-integrated angular weight of dcs.hh:913-934, each operation rounded as in
// the reference: both of its differences cancel as q grows (a mean error of 230
// ulp above 1 TeV), and with a rcp(b) for the quotients the mean error was 12%
// larger.  VALUE = false, where only finiteness is asked: a rcp(b).
template <bool VALUE>
__device__ __forceinline__ double soft_ratio(double K, double q, double mass) {
    const auto quot = [](double a, double b) { return VALUE ? ol_qdiv(a, b) : a * ol_rcp(b); };
    const double E = x_add(K, mass);
    const double m02 = 0.4;
    const double q2 = x_mul(q, q);
    const double tmax = x_mul(1.876544, q);
    const double tmin = quot(x_mul(x_mul(q2, mass), mass), x_mul(E, x_sub(E, q)));
    // the poles (q^2 = m02)
    const double b1 = quot(1., x_sub(1., x_div(q2, m02)));
    const double c1 = quot(1., x_sub(1., x_div(m02, q2)));
    double L1 = x_mul(b1, ol_log(quot(x_add(q2, tmax), x_add(q2, tmin))));
    double L2 = x_mul(c1, ol_log(quot(x_add(m02, tmax), x_add(m02, tmin))));
    const double I0 = x_sub(x_sub(ol_log(quot(tmax, tmin)), L1), L2);
    L1 = x_mul(L1, q2);
    L2 = x_mul(L2, m02);
    const double I1 = x_add(L1, L2);
    L1 = x_mul(L1, q2);
    L2 = x_mul(L2, m02);
    const double I2 = x_sub(x_sub(x_mul(x_sub(tmax, tmin), x_add(x_mul(b1, q2), x_mul(c1, m02))), L1), L2);
    return quot(x_sub(x_mul(I1, tmax), I2),
                x_mul(x_mul(x_sub(x_mul(I0, tmax), I1), K), x_add(K, x_mul(2., mass))));
}

// dcs.hh:874-899 in the reference's operation order.
__device__ __forceinline__ double soft_ionisation(double K, const noa_dcs_consts &c) {
    const double mass = c.mass;
    const double p2 = x_mul(K, x_add(K, x_mul(2., mass)));
    const double E = x_add(K, mass);
    const double Wmax = x_div(x_mul(x_mul(2., ME), p2), x_add(x_mul(mass, mass), x_mul(ME, x_add(ME, x_mul(2., E)))));
    const double W0 = x_div(x_mul(2., p2), ME);
    const double mu_max = x_div(Wmax, W0);
    double mu3 = x_div(x_mul(K, NOA_X_FRACTION), W0);
    if (mu3 > mu_max)
        mu3 = mu_max;
    const double mu2 = x_div(x_mul(0.62, c.I), W0);
    if (mu2 >= mu3)
        return 0.;
    const double a0 = x_div(x_mul(0.5, W0), p2);
    const double a1 = x_div(-1., Wmax);
    const double a2 = x_div(x_mul(E, E), x_mul(W0, p2));
    const double cs0 = x_div(1.535336E-05, c.A);
    const double bracket = x_add(x_add(x_mul(x_mul(0.5, a0), x_sub(x_mul(mu3, mu3), x_mul(mu2, mu2))),
                                       x_mul(a1, x_sub(mu3, mu2))),
                                 x_mul(a2, log(x_div(mu3, mu2))));
    return x_mul(x_mul(x_mul(2., cs0), c.Zd), bracket);
}

// Node i of the rule for kinetic energy K: nu and q (numerics.hh:84-86, dcs.hh:910-911).
__device__ __forceinline__ void soft_node(double K, int i, const SoftParams &p, double &nu, double &q) {
    const double t = x_add(p.lb, x_mul(p.h, fpconv::f64i(i / 6) + kGL6X[i % 6]));
    nu = x_mul(NOA_X_FRACTION, lean_exp(t));
    q = x_mul(nu, K);
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS, i_ctas(THREADS))
    soft_scattering_kernel(const SoftParams p, const noa_dcs_consts c) {
    constexpr int I_BATCH = i_batch(THREADS);
    __shared__ double vals[S_KMAX * S_NODES];
    __shared__ int qS[queue_capacity(I_BATCH, THREADS)];
    __shared__ QuadSmem<NOA_DCS_PROC_PHOTO, I_BATCH> quad;
    __shared__ double sK[S_KMAX];
    __shared__ int warp_tot[THREADS / 32];
    __shared__ int tile_open;
    const int pairs = p.kpt * S_NODES;
    const int64_t tiles = (p.n + p.kpt - 1) / p.kpt;

    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t k0 = tile * p.kpt;
        if ((int)threadIdx.x < p.kpt) {
            const int64_t ki = k0 + threadIdx.x;
            sK[threadIdx.x] = ki < p.n ? p.K[ki] : 1.;
        }
        __syncthreads();
        int qn = 0;
        for (int base = 0;; base += THREADS) {
            const bool more = base < pairs;  // block-uniform
            if (more) {
                const int slot = base + threadIdx.x;
                bool open = false;
                if (slot < pairs) {
                    const int kk = slot / S_NODES, i = slot - kk * S_NODES;
                    vals[slot] = 0.;
                    if (k0 + kk < p.n) {
                        const double K = sK[kk];
                        double nu, q;
                        soft_node(K, i, p, nu, q);
                        open = photo_live(K, q, c);
                        // closed: the reference adds 0 * ratio * nu, which is 0 (of either sign, which
                        // the node sum cannot tell apart) unless the ratio is not finite
                        if (!open && !isfinite(soft_ratio<false>(K, q, c.mass)))
                            vals[slot] = __longlong_as_double(0x7FF8000000000000LL);   // NaN, as 0 * inf
                    }
                }
                const int pos = qn + block_scan<THREADS>(open ? 1 : 0, warp_tot, &tile_open);
                if (open)
                    qS[pos] = slot;
                __syncthreads();
                qn += tile_open;
            }
            // one call site of the evaluation, as in the recoil integrals
            while (qn >= I_BATCH || (!more && qn > 0)) {
                const int take = qn < I_BATCH ? qn : I_BATCH;
                const int first = qn - take;
                double nu = 0.;  // of this thread's own pair
                quad_batch<NOA_DCS_PROC_PHOTO, THREADS>(
                    quad, take, c,
                    [&](int e, double &K, double &q) {
                        const int sl = qS[first + e], kk = sl / S_NODES;
                        K = sK[kk];
                        soft_node(K, sl - kk * S_NODES, p, nu, q);
                    },
                    [&](int e, double d) {
                        const int sl = qS[first + e], kk = sl / S_NODES;
                        const double K = sK[kk];
                        const double f = x_mul(x_mul(d, soft_ratio<true>(K, x_mul(nu, K), c.mass)), nu);
                        vals[sl] = x_mul(x_mul(f, p.h), kGL6W[(sl - kk * S_NODES) % 6]);
                    });
                qn -= take;
                __syncthreads();
            }
            if (!more)
                break;
        }
        __syncthreads();
        for (int kk = threadIdx.x >> 5; kk < p.kpt && k0 + kk < p.n; kk += THREADS / 32) {
            const double s = warp_node_sum(vals + kk * S_NODES, S_NODES);
            if ((threadIdx.x & 31) == 0)
                p.out[k0 + kk] = x_add(soft_ionisation(sK[kk], c), x_mul(2., s));
        }
        __syncthreads();
    }
}

static int sm_count() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 1;
}

} // namespace noa_dcs

using namespace noa_dcs;

namespace {

// Energies per tile: one while the call has fewer than 20 tiles an SM, then
// up to `most`.
int energies_per_tile(int64_t n, int64_t sms, int most) {
    const int64_t k = n / (sms * 20);
    return (int)(k < 1 ? 1 : (k > most ? most : k));
}

// The width for n energies of `nodes` nodes.  Up to one an SM a CTA has the SM
// for itself: the (pair, node) rounds of the quadrature processes shrink up to
// 1024 threads (pair production / photonuclear, 146 energies of 180 nodes:
// 54.9 / 70.0 us at 128 threads, 34.0 / 46.4 at 256, 27.3 / 39.3 at 512, 26.8 /
// 36.4 at 1024), while bremsstrahlung, ionisation and soft scattering, which
// wait for one or two rounds of usual node counts, are as fast at 256 as above
// (9.8, 10.1 and 26.3 us).  Up to two an SM both are resident at 256 (304
// energies: 43.3 / 63.0 us against 60.5 / 80.9 at 128 and 51.3 / 69.6 at 1024);
// a quadrature's batch of 192 leaves room for 4 KB of node values there.
// Above, 128 threads leave room for five (456 energies: 14.5 us of
// bremsstrahlung against 19.8 at 256).
constexpr int I_MID_NODES = 512;
int integral_width(bool quadrature, int nodes, int64_t n, int64_t sms) {
    const bool few = nodes <= I_MID_NODES;
    if (n <= sms)
        return quadrature || !few ? I_WIDE : I_MID;
    return n <= 2 * sms && (few || !quadrature) ? I_MID : I_NARROW;
}

template <int THREADS>
cudaError_t launch_recoil(int process, const IntegralParams &p, const noa_dcs_consts &c, cudaStream_t stream) {
    const int64_t tiles = (p.n + p.kpt - 1) / p.kpt;
    const int grid = (int)(tiles < (1 << 30) ? tiles : (1 << 30));
    const size_t smem = sizeof(double) * (size_t)(p.kpt * p.nodes);
    switch (process) {
    case NOA_DCS_PROC_BREMS:
        recoil_integral_kernel<NOA_DCS_PROC_BREMS, THREADS><<<grid, THREADS, smem, stream>>>(p, c);
        break;
    case NOA_DCS_PROC_PPROD:
        recoil_integral_kernel<NOA_DCS_PROC_PPROD, THREADS><<<grid, THREADS, smem, stream>>>(p, c);
        break;
    case NOA_DCS_PROC_PHOTO:
        recoil_integral_kernel<NOA_DCS_PROC_PHOTO, THREADS><<<grid, THREADS, smem, stream>>>(p, c);
        break;
    case NOA_DCS_PROC_ION:
        recoil_integral_kernel<NOA_DCS_PROC_ION, THREADS><<<grid, THREADS, smem, stream>>>(p, c);
        break;
    default:
        return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

} // namespace

cudaError_t noa_dcs_launch_recoil_integral(int process, int moment, const double *K, double *out, int64_t n,
                                           double xlow, int min_points, const noa_dcs_consts *c,
                                           cudaStream_t stream) {
    if (n <= 0)
        return cudaSuccess;
    IntegralParams p;
    p.K = K;
    p.out = out;
    p.n = n;
    p.xlow = xlow;
    p.n_itv = (min_points + 5) / 6;
    p.nodes = 6 * p.n_itv;
    if (p.nodes > I_PAIRS || p.nodes < 6)
        return cudaErrorInvalidValue;
    const int64_t sms = sm_count();
    const int most = p.nodes >= I_PAIRS / 2 ? 1 : I_PAIRS / 2 / p.nodes;
    p.kpt = energies_per_tile(n, sms, most < I_KMAX ? most : I_KMAX);
    p.moment = moment;
    switch (integral_width(is_quad(process), p.nodes, n, sms)) {
    case I_WIDE:
        return launch_recoil<I_WIDE>(process, p, *c, stream);
    case I_MID:
        return launch_recoil<I_MID>(process, p, *c, stream);
    default:
        return launch_recoil<I_NARROW>(process, p, *c, stream);
    }
}

cudaError_t noa_dcs_launch_soft_scattering(const double *K, double *out, int64_t n, const noa_dcs_consts *c,
                                           cudaStream_t stream) {
    if (n <= 0)
        return cudaSuccess;
    SoftParams p;
    p.K = K;
    p.out = out;
    p.n = n;
    p.lb = log(1E-06);                // dcs.hh:905
    p.h = (0. - p.lb) / (double)17u;  // numerics.hh:80-81, n_itv = ceil(100 / 6)
    const int64_t sms = sm_count();
    p.kpt = energies_per_tile(n, sms, S_KMAX);
    const int64_t tiles = (n + p.kpt - 1) / p.kpt;
    const int grid = (int)(tiles < (1 << 30) ? tiles : (1 << 30));
    if (integral_width(false, S_NODES, n, sms) == I_MID)
        soft_scattering_kernel<I_MID><<<grid, I_MID, 0, stream>>>(p, *c);
    else
        soft_scattering_kernel<I_NARROW><<<grid, I_NARROW, 0, stream>>>(p, *c);
    return cudaGetLastError();
}
