// cl_surrogate.cu — events from the learned light-response surrogate.
//
// The surrogate (cl_mlp.cu) maps an emission point to, per SiPM, the
// probability that a photon emitted there is detected by that SiPM and the
// mean and log standard deviation of the detected photons' transit times.
// For a 511 keV event the deposits ("sites") that the surrogate can be
// trusted with are sampled here instead of transported:
//
//   * surrogate_combine: the K ensemble members' outputs -> ensemble-mean
//     probabilities (times the PDE), transit-time mean and sigma, the members'
//     relative spread, and a fallback flag (spread above a threshold, the
//     site within a distance of a wrapped face, or detection probabilities
//     summing to 1 or more) that sends the site to the plain Monte Carlo;
//   * surrogate_sample: per unflagged site, the N emitted photons are split
//     over the SiPMs multinomially by a chain of conditional binomial draws
//     (n_j ~ Bin(N - sum_{i<j} n_i, p_j / (1 - sum_{i<j} p_i))), and each
//     SiPM's first-hit time is drawn exactly as the minimum of its n_j arrival
//     times, each an exponential emission delay (decay time tau) plus a
//     Gaussian transit time: the minimum's CDF is 1 - (1 - F)^n_j with F the
//     exponentially modified Gaussian CDF, inverted by safeguarded Newton.
//
// Binomial variates: inversion for n*p < 10, otherwise Hormann's BTRD
// (W. Hormann, "The generation of binomial random variates", J. Statist.
// Comput. Simul. 46 (1993) 101-110), both in Float64.  Uniforms come from
// Philox4x32-10 keyed with the event seed, counter (site lo, site hi, block,
// 0x53555247): a stream domain disjoint from the transport's photon streams
// (whose fourth counter word is 0).
//
// Every loop is bounded; a budget that runs out sets bit 2 of the error word
// and the site's remaining draws fall back to the mean.  A site whose segment
// id lies outside the maps is skipped and sets bit 3.
#include <cmath>
#include <cstdint>

#include <cuda_runtime.h>

#include "../../include/crysplight_cuda.h"
#include "cl_device.cuh"
#include "cl_surrogate.cuh"

namespace cl {
namespace sur {

constexpr uint32_t STREAM_TAG = 0x53555247u;   // "SURG": a site's binomial chain
constexpr uint32_t TIME_TAG = 0x53555254u;     // "SURT": a (site, SiPM) first-hit time
constexpr int CELLS = 64;                      // SiPMs of the readout grid
constexpr unsigned SAMPLER_BUDGET_BIT = 4u;

// Float64 uniforms in (0, 1) from one Philox stream.
struct Uni {
    uint32_t lo, hi, block, k0, k1;
    uint32_t buf[4];
    int left;
    __device__ void init(uint64_t stream, uint32_t key0, uint32_t key1)
    {
        lo = (uint32_t)stream; hi = (uint32_t)(stream >> 32); block = 0; k0 = key0; k1 = key1; left = 0;
    }
    __device__ double next()
    {
        if (left == 0) {
            const uint4 o = philox4x32_10(make_uint4(lo, hi, block, STREAM_TAG), k0, k1);
            block += 1u;
            buf[0] = o.x; buf[1] = o.y; buf[2] = o.z; buf[3] = o.w;
            left = 4;
        }
        const uint32_t x = buf[4 - left];
        left -= 1;
        return ((double)x + 0.5) * 0x1p-32;
    }
};

// Stirling-series remainder fc(k) = log(k!) - [(k + 1/2) log(k + 1) - (k + 1) + log(2 pi)/2].
__device__ double stirling_fc(int64_t k)
{
    const double N = (double)k + 1.0;
    if (k < 10) return lgamma(N) - (N - 0.5) * log(N) + N - 0.91893853320467274178;
    const double r = 1.0 / N, r2 = r * r;
    return (1.0 / 12.0 - (1.0 / 360.0 - (1.0 / 1260.0) * r2) * r2) * r;
}

// Inversion, n * p < 10, p <= 1/2 (sequential search from 0).
__device__ int64_t binom_inversion(int64_t n, double p, Uni& U, unsigned& bad)
{
    const double q = 1.0 - p, s = p / q, a = (double)(n + 1) * s;
    const double r0 = exp((double)n * log1p(-p));
    for (int attempt = 0; attempt < 64; ++attempt) {
        double u = U.next(), r = r0;
        int64_t x = 0;
        for (;;) {
            if (u <= r) return x;
            u -= r;
            ++x;
            if (x > n || x > 200) break;        // round-off tail: draw again
            r *= a / (double)x - s;
        }
    }
    bad |= SAMPLER_BUDGET_BIT;
    return (int64_t)((double)n * p + 0.5);
}

// BTRD, n * p >= 10, p <= 1/2.
__device__ int64_t binom_btrd(int64_t n, double p, Uni& U, unsigned& bad)
{
    const double q = 1.0 - p;
    const double np = (double)n * p, npq = np * q, spq = sqrt(npq);
    const int64_t m = (int64_t)floor((double)(n + 1) * p);
    const double r = p / q, nr = (double)(n + 1) * r;
    const double b = 1.15 + 2.53 * spq;
    const double a = -0.0873 + 0.0248 * b + 0.01 * p;
    const double c = np + 0.5;
    const double alpha = (2.83 + 5.1 / b) * spq;
    const double vr = 0.92 - 4.2 / b;
    const double urvr = 0.86 * vr;
    for (int it = 0; it < 1000; ++it) {
        double v = U.next(), u;
        if (v <= urvr) {
            u = v / vr - 0.43;
            return (int64_t)floor((2.0 * a / (0.5 - fabs(u)) + b) * u + c);
        }
        if (v >= vr) {
            u = U.next() - 0.5;
        } else {
            u = v / vr - 0.93;
            u = copysign(0.5, u) - u;
            v = U.next() * vr;
        }
        const double us = 0.5 - fabs(u);
        const double kd = floor((2.0 * a / us + b) * u + c);
        if (kd < 0.0 || kd > (double)n) continue;
        const int64_t k = (int64_t)kd;
        v = v * alpha / (a / (us * us) + b);
        const int64_t km = k > m ? k - m : m - k;
        if (km <= 15) {
            double f = 1.0;
            if (m < k) {
                for (int64_t i = m + 1; i <= k; ++i) f *= nr / (double)i - r;
            } else if (m > k) {
                for (int64_t i = k + 1; i <= m; ++i) v *= nr / (double)i - r;
            }
            if (v <= f) return k;
            continue;
        }
        v = log(v);
        const double kmd = (double)km;
        const double rho = (kmd / npq) * (((kmd / 3.0 + 0.625) * kmd + 1.0 / 6.0) / npq + 0.5);
        const double t = -kmd * kmd / (2.0 * npq);
        if (v < t - rho) return k;
        if (v > t + rho) continue;
        const double nm = (double)(n - m + 1);
        const double h = ((double)m + 0.5) * log(((double)m + 1.0) / (r * nm)) + stirling_fc(m) +
                         stirling_fc(n - m);
        const double nk = (double)(n - k + 1);
        if (v <= h + (double)(n + 1) * log(nm / nk) + ((double)k + 0.5) * log(nk * r / ((double)k + 1.0)) -
                     stirling_fc(k) - stirling_fc(n - k))
            return k;
    }
    bad |= SAMPLER_BUDGET_BIT;
    return (int64_t)(np + 0.5);
}

__device__ int64_t binomial(int64_t n, double p, Uni& U, unsigned& bad)
{
    if (n <= 0 || !(p > 0.0)) return 0;
    if (p >= 1.0) return n;
    const bool flip = p > 0.5;
    const double pp = flip ? 1.0 - p : p;
    const int64_t k = ((double)n * pp < 10.0) ? binom_inversion(n, pp, U, bad) : binom_btrd(n, pp, U, bad);
    return flip ? n - k : k;
}

// Exponentially modified Gaussian: X = E + T, E ~ Exp(rate lam), T ~ N(mu, sigma^2),
// in the standardised variable z = (t - mu) / sigma with ls = lam * sigma.
// Returns F(t) and sets *dens to the density f(t).
// Both terms carry exp(-z^2/2) where it would otherwise under/overflow
// (erfcx(x) = exp(x^2) erfc(x)).
__device__ double emg_cdf(double z, double ls, double lam, double* dens)
{
    constexpr double R2 = 0.70710678118654752440;
    const double w = z - ls;
    double phi_z, term2;
    if (w < 0.0) {
        term2 = 0.5 * exp(-0.5 * z * z) * erfcx(-w * R2);
    } else {
        term2 = 0.5 * exp(-ls * z + 0.5 * ls * ls) * erfc(-w * R2);
    }
    if (z < 0.0) phi_z = 0.5 * exp(-0.5 * z * z) * erfcx(-z * R2);
    else phi_z = 0.5 * erfc(-z * R2);
    *dens = lam * term2;            // density per unit t
    return phi_z - term2;
}

// Minimum of k >= 1 independent EMG(mu, sigma, tau) arrival times, by
// inverting P(min <= t) = 1 - (1 - F(t))^k at the uniform u in (0, 1).
__device__ double emg_min_u(int64_t k, double mu, double sigma, double tau, double u, unsigned& bad)
{
    const double lu = log(u) / (double)k;       // log of the survival level, < 0
    const double y = -expm1(lu);                // target F(t) in (0, 1)
    if (!(tau > 0.0)) return mu + sigma * normcdfinv(y);
    if (!(sigma > 0.0)) return mu - tau * lu;   // pure exponential: F = 1 - exp(-(t - mu)/tau)
    const double lam = 1.0 / tau, ls = lam * sigma;
    // bracket in z: F(lo) < y <= F(hi)
    double lo = -40.0, hi = 12.0 + (-tau * lu) / sigma + 0.5 * tau / sigma;
    double dens = 0.0;
    for (int g = 0; g < 64 && emg_cdf(hi, ls, lam, &dens) < y; ++g) hi = 2.0 * hi + 1.0;
    double z = fmin(fmax((-tau * lu) / sigma, lo), hi);
    for (int it = 0; it < 100; ++it) {
        const double F = emg_cdf(z, ls, lam, &dens) - y;
        if (F < 0.0) lo = z; else hi = z;
        const double fz = dens * sigma;            // dF/dz
        double zn = (fz > 0.0) ? z - F / fz : 0.5 * (lo + hi);
        if (!(zn > lo && zn < hi)) zn = 0.5 * (lo + hi);
        if (fabs(zn - z) < 1e-9 * fmax(1.0, fabs(z)) || hi - lo < 1e-9 * fmax(1.0, fabs(z)))
            return mu + sigma * zn;
        z = zn;
    }
    bad |= SAMPLER_BUDGET_BIT;
    return mu + sigma * z;
}

__device__ double emg_min(int64_t k, double mu, double sigma, double tau, Uni& U, unsigned& bad)
{
    return emg_min_u(k, mu, sigma, tau, U.next(), bad);
}

// The uniform of the first-hit time of SiPM c at site i: word 0 of its own
// Philox block (counter (site lo, site hi, c, "SURT")), disjoint from the
// site's binomial stream and from the transport's photon streams.
__device__ __forceinline__ double time_uniform(int64_t i, int c, uint32_t k0, uint32_t k1)
{
    const uint4 o = philox4x32_10(make_uint4((uint32_t)i, (uint32_t)((uint64_t)i >> 32), (uint32_t)c, TIME_TAG),
                                  k0, k1);
    return ((double)o.x + 0.5) * 0x1p-32;
}

// Warp-cooperative: each lane runs the binomial chain of one site (the
// chain is sequential over the SiPMs), recording the hit counts in shared
// memory; then the warp's lanes share out the first-hit times of all
// (site, SiPM) pairs that were hit, which cost far more than the chain (a
// safeguarded Newton inversion in Float64 each) and which thread-per-site
// code would leave to the lanes of the sites with the most hit SiPMs.  Each
// pair's time comes from its own uniform (time_uniform), so the result does
// not depend on which lane draws it.  Eight CTAs of 128 threads per SM
// (64 registers; the Float64 special functions' latency needs the warps more
// than the spilled registers cost).
//
// A warp takes `sites` sites at a time, the fewest (a power of two) with which
// all warps are resident at once: the chain is a latency of 64 dependent draws
// however few lanes run it, and the times are shared out over all lanes anyway.
// 2,800 sites: 1451 us with 32 per warp, 951 / 642 / 509 / 444 / 410 with 16 / 8
// / 4 / 2 / 1; 28,000: 1725, 1545 / 1550 / 2320 (two waves) with 16 / 8 / 4.
constexpr int SAMPLE_WARPS = 4, SAMPLE_CTAS = 8;
__global__ void __launch_bounds__(32 * SAMPLE_WARPS, SAMPLE_CTAS) surrogate_sample(const SurSampleArgs A, int sites)
{
    __shared__ uint16_t s_k[SAMPLE_WARPS][CELLS][32];   // hit counts of the warp's sites, by SiPM
    __shared__ uint32_t s_mask[SAMPLE_WARPS][CELLS];    // lanes whose site hit the SiPM
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cells = A.cells;                          // <= CELLS (launcher)
    const int64_t nwarps = (int64_t)gridDim.x * SAMPLE_WARPS;
    unsigned bad = 0;
    unsigned long long ph = 0, det = 0;
    for (int64_t i0 = ((int64_t)blockIdx.x * SAMPLE_WARPS + wib) * sites; i0 < A.n; i0 += nwarps * sites) {
        // ---- the binomial chain of this lane's site ----
        const int64_t i = i0 + lane;
        int64_t left = 0, base = 0;
        if (lane < sites && i < A.n && !(A.flag && A.flag[i])) {
            left = A.photons[i];
            if (left > 0) {
                const int32_t sg = A.seg[i];
                if (sg < 0 || (int64_t)sg >= A.n_seg) { bad |= 8u; left = 0; }
                else { base = (int64_t)sg * cells; ph += (unsigned long long)left; }
            } else {
                left = 0;
            }
        }
        Uni U;
        U.init((uint64_t)i, A.k0, A.k1);
        const float* p = A.p + i * cells;
        double mass = 1.0;                          // probability not yet assigned
        for (int c = 0; c < cells; ++c) {
            int64_t k = 0;
            if (left > 0) {
                const double pc = (double)p[c];
                const double pcond = mass > 0.0 ? fmin(fmax(pc / mass, 0.0), 1.0) : 1.0;
                mass -= pc;
                k = binomial(left, pcond, U, bad);
                if (k > 0) {
                    left -= k;
                    det += (unsigned long long)k;
                    atomicAdd(A.maps + base + c, (uint32_t)k);
                    if (k > 65535) {
                        // beyond the shared counts' range: this lane draws its time now
                        const double t = emg_min_u(k, (double)A.tmean[i * cells + c], (double)A.tsig[i * cells + c],
                                                   (double)A.tau, time_uniform(i, c, A.k0, A.k1), bad);
                        atomicMin(A.keys + base + c, float_key((float)((double)A.t0[i] + t)));
                        k = 0;
                    }
                }
            }
            s_k[wib][c][lane] = (uint16_t)k;
            const unsigned m = __ballot_sync(0xffffffffu, k > 0);
            if (lane == 0) s_mask[wib][c] = m;
        }
        __syncwarp();
        // ---- the first-hit times of every (site, SiPM) pair hit, shared out ----
        int total = 0;
        for (int c = 0; c < cells; ++c) total += __popc(s_mask[wib][c]);
        int c = 0, before = 0;                      // items of SiPMs < c
        for (int item = lane; item < total; item += 32) {
            while (item >= before + __popc(s_mask[wib][c])) { before += __popc(s_mask[wib][c]); ++c; }
            const unsigned m = s_mask[wib][c];
            const int sl = (int)__fns(m, 0u, item - before + 1);     // the site's lane
            const int64_t is = i0 + sl;
            const int64_t kk = s_k[wib][c][sl];
            const double t = emg_min_u(kk, (double)A.tmean[is * cells + c], (double)A.tsig[is * cells + c],
                                       (double)A.tau, time_uniform(is, c, A.k0, A.k1), bad);
            atomicMin(A.keys + (int64_t)A.seg[is] * cells + c, float_key((float)((double)A.t0[is] + t)));
        }
        __syncwarp();
    }
    if (A.stats) {
        // one pair of atomics per warp
        for (int o = 16; o > 0; o >>= 1) {
            ph += __shfl_down_sync(0xffffffffu, ph, o);
            det += __shfl_down_sync(0xffffffffu, det, o);
        }
        if ((threadIdx.x & 31) == 0 && (ph | det)) {
            atomicAdd(A.stats, ph);
            atomicAdd(A.stats + 1, det);
        }
    }
    if (bad) atomicOr(A.err, bad);
}

// Ensemble reduction: one warp per site, two SiPMs per lane, all outputs of up
// to COMBINE_BATCH members requested before the first is used (members beyond
// them in further batches), no CTA barrier.  The bound is the members' outputs
// from HBM or L2 (768 bytes per site and member); with 64 threads per site,
// three loads in flight per thread and two barriers per site the kernel waited
// on memory: 42,000 sites x 5 members 111 -> 68 us, 1 member 45 -> 43, 7 members
// 142 -> 88 (a batch that always loads five rows, the last one again and again:
// 70, 47 and 98).
struct CombineArgs {
    const float* raw;        // [K][n][3 * cells] standardised member outputs
    int32_t K;
    int64_t n;
    const float* y_mean;     // [3 * cells]
    const float* y_std;      // [3 * cells]
    const float* xyz;        // mm, row site[i] (i where site is null)
    const int32_t* site;     // row of the sites' arrays of each row i (may be null)
    const float* direct;     // [n][CELLS] first-pass probabilities added to the members' (may be null)
    float L0, L1, L2;
    int32_t front_wrapped;
    float pde, spread_max, wall_min_mm;
    float* p;
    float* tmean;
    float* tsig;
    float* spread;
    uint8_t* flag;
};

constexpr int COMBINE_WARPS = 8;
constexpr int COMBINE_BATCH = 5;

__global__ void __launch_bounds__(32 * COMBINE_WARPS) surrogate_combine(const CombineArgs A)
{
    const int lane = threadIdx.x & 31;
    float mean[3][2], std[3][2];                 // per output kind and SiPM
#pragma unroll
    for (int o = 0; o < 3; ++o)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            mean[o][q] = A.y_mean[o * CELLS + 32 * q + lane];
            std[o][q] = A.y_std[o * CELLS + 32 * q + lane];
        }
    const double invK = 1.0 / (double)A.K;
    const int64_t stride = (int64_t)gridDim.x * COMBINE_WARPS;
    for (int64_t i = (int64_t)blockIdx.x * COMBINE_WARPS + (threadIdx.x >> 5); i < A.n; i += stride) {
        const int64_t to = A.site ? A.site[i] : i;
        double sum_p[2] = {0.0, 0.0}, sum_p2[2] = {0.0, 0.0}, sum_t[2] = {0.0, 0.0}, sum_l[2] = {0.0, 0.0};
        float dir[2] = {0.f, 0.f};
        if (A.direct) {
            dir[0] = A.direct[i * CELLS + lane];
            dir[1] = A.direct[i * CELLS + 32 + lane];
        }
        for (int k0 = 0; k0 < A.K; k0 += COMBINE_BATCH) {
            float v[COMBINE_BATCH][3][2];
#pragma unroll
            for (int k = 0; k < COMBINE_BATCH; ++k) {
                if (k0 + k >= A.K) break;
                const float* row = A.raw + ((int64_t)(k0 + k) * A.n + i) * (3 * CELLS) + lane;
#pragma unroll
                for (int o = 0; o < 3; ++o)
#pragma unroll
                    for (int q = 0; q < 2; ++q) v[k][o][q] = __ldcs(row + o * CELLS + 32 * q);
            }
#pragma unroll
            for (int k = 0; k < COMBINE_BATCH; ++k) {
                if (k0 + k >= A.K) break;
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const double pk = exp((double)v[k][0][q] * std[0][q] + mean[0][q]);
                    sum_p[q] += pk;
                    sum_p2[q] += pk * pk;
                    sum_t[q] += (double)v[k][1][q] * std[1][q] + mean[1][q];
                    sum_l[q] += (double)v[k][2][q] * std[2][q] + mean[2][q];
                }
            }
        }
        double a[2], b[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const double pr = sum_p[q] * invK;
            const double var = fmax(sum_p2[q] * invK - pr * pr, 0.0);
            // the first-pass term is the same for every member: it adds to the
            // mean and to the total the spread is relative to, not to the spread
            const double pm = pr + (A.direct ? (double)dir[q] : 0.0);
            a[q] = sqrt(var);
            b[q] = pm;
            const int64_t at = to * CELLS + 32 * q + lane;
            A.p[at] = (float)(pm * (double)A.pde);
            A.tmean[at] = (float)(sum_t[q] * invK);
            A.tsig[at] = (float)exp(sum_l[q] * invK);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                a[q] += __shfl_down_sync(0xffffffffu, a[q], o);
                b[q] += __shfl_down_sync(0xffffffffu, b[q], o);
            }
        if (lane == 0) {
            const double num = a[0] + a[1];
            const double den = b[0] + b[1];
            const float spr = (float)(num / fmax(den, 1e-30));
            const float x = A.xyz[3 * to], y = A.xyz[3 * to + 1], z = A.xyz[3 * to + 2];
            float d = fminf(fminf(x, A.L0 - x), fminf(y, A.L1 - y));
            if (A.front_wrapped) d = fminf(d, z);
            uint8_t f = 0;
            if (!(spr <= A.spread_max)) f |= 1u;
            if (d < A.wall_min_mm) f |= 2u;
            if (!(den * (double)A.pde < 0.999)) f |= 4u;   // not a probability split: Monte Carlo
            A.spread[to] = spr;
            A.flag[to] = f;
        }
    }
}

// First-pass light (the analytic part of the light response): the
// probability that a photon emitted isotropically at a site reaches the
// readout face z = Lz without a bulk interaction and crosses into SiPM c
// there, at PDE 1.  A photon leaving at polar angle theta from the face normal
// travels h / cos(theta) (h = Lz - z) and survives absorption and Rayleigh
// scattering with probability exp(-mu h / cos theta), mu = 1/abs_len +
// 1/rayleigh (the competition of the two exponential path lengths against
// the face distance); the face transmits it with probability 1 - R(cos
// theta) (the same Fresnel coefficients, total internal reflection beyond
// the critical angle); it lands on the circle of radius rho = h tan(theta)
// about the site's projection, uniformly in azimuth, and is detected by the
// SiPM whose pixel contains the landing point (pixel c = j nx + i for
// floor(x / pitch) = i, the last column and row reaching the face edge;
// landing points off the face belong to a side wall first and are not
// first-pass light).  So
//     D_c = 1/(4 pi) int_0^theta_max (1 - R) exp(-mu h / cos theta) sin theta
//           * (arc of the circle inside pixel c) d theta,
// with the arcs exact (intersections of the circle with the pixel's column
// and row strips) and theta by composite Gauss-Legendre quadrature (8 panels
// of 8 nodes up to the critical angle).  The nodes' contributions are summed as
// 2^-40 fixed-point integers, so the result does not depend on the order they
// are added in: a site's term is the same bits in any batch.
//
// One warp per site.  First every lane takes two nodes and writes the angles at
// which its circle crosses the edges of the pixel columns and rows it reaches
// (arc cosines and sines: once per edge, not four per pixel; for the columns or
// rows of grids wider than DIRECT_TABULATED, at each use).  A pixel is
// crossed by a contiguous range of nodes, because the radii increase; the
// (pixel, node) items of all 64 pixels are then shared out evenly over the
// lanes (near the face one pixel has all 64 nodes).  The bound is instruction
// issue.  A lane per pixel kept 11 of 32 lanes active and took 344 us; a thread per
// node that evaluated four angles and one shared-memory atomic per pixel of its
// circle's bounding box, four sites per CTA behind common barriers, issued on
// 49% of its cycles: 42,000 sites 404 -> 179 us.
// The rest of the light response (reflections, scattering) varies slowly
// over the SiPM plane; a surrogate trained on it learns what the first-pass
// term's sharp pixel edges would otherwise ask of it.
namespace {
// 8-point Gauss-Legendre nodes and weights on [-1, 1] (positive half)
__constant__ double c_gl_x[4] = {0.1834346424956498, 0.5255324099163290, 0.7966664774136267, 0.9602898564975363};
__constant__ double c_gl_w[4] = {0.3626837833783620, 0.3137066458778873, 0.2223810344533745, 0.1012285362903763};
}

struct DirectArgs {
    const float* xyz;        // mm, row site[i] (i where site is null)
    const int32_t* site;     // (may be null)
    int64_t n;
    float L0, L1, L2;
    float n1, n2, mu;        // crystal and coupling indices, attenuation 1/mm
    float pitch;
    int32_t nx, ny;
    float* out;              // [n][CELLS]
};

constexpr int DIRECT_NODES = 64;
constexpr double DIRECT_FIX = 1099511627776.0;   // 2^40
constexpr int DIRECT_WARPS = 8;
constexpr int DIRECT_STRIDE = DIRECT_NODES + 1;  // floats per edge (odd: lanes at different edges on different banks)
// Columns (rows) up to which their edges' angles are tabulated.  A wider grid's
// table takes the shared memory that other warps need (64 x 1: 8 warps per SM):
// 42,000 sites on 64 x 1 pixels 370 us tabulated and 102 with the columns' angles
// taken per item (268 by the kernel with a thread per node), on 32 x 2 246 and 175
// (322).  A narrower one's is read often enough: 16 x 4 209 and 256.
constexpr int DIRECT_TABULATED = 16;
constexpr int DIRECT_MAX_EDGES = 22;             // 16 x 4 pixels: 17 + 5
constexpr float TWO_PI_ARC = 6.283185307179586f;

// Shared floats of a warp: the angles of the tabulated edges, per node its weight
// (double), radius, inverse radius and bounding box, per pixel its sum (64 bits),
// first item and first node.
__host__ __device__ constexpr int direct_warp_floats(int edges)
{
    return edges * DIRECT_STRIDE + edges % 2 + 5 * DIRECT_NODES + 4 * CELLS;
}

// The angles at which a circle crosses a column's or a row's edge, for the
// quotient of the edge's distance from the site and the radius.
__device__ __forceinline__ float column_angle(float v) { return acosf(fminf(fmaxf(v, -1.0f), 1.0f)); }
__device__ __forceinline__ float row_angle(float v) { return asinf(fminf(fmaxf(v, -1.0f), 1.0f)); }

template <bool XTAB, bool YTAB>
__global__ void __launch_bounds__(32 * DIRECT_WARPS) surrogate_direct(const DirectArgs A)
{
    extern __shared__ __align__(16) float s_direct[];
    __shared__ double s_w[DIRECT_NODES], s_c[DIRECT_NODES];
    __shared__ float s_tan[DIRECT_NODES];
    const int lane = threadIdx.x & 31;
    const int nx = A.nx, ny = A.ny;
    const int x_edges = XTAB ? nx + 1 : 0, edges = x_edges + (YTAB ? ny + 1 : 0);
    float* const aa = s_direct + (threadIdx.x >> 5) * direct_warp_floats(edges);   // [edge][node]
    float* const ba = aa + x_edges * DIRECT_STRIDE;
    double* const wt = reinterpret_cast<double*>(aa + edges * DIRECT_STRIDE + edges % 2);   // weight x 2^40
    unsigned long long* const acc = reinterpret_cast<unsigned long long*>(wt + DIRECT_NODES);
    float* const rad = reinterpret_cast<float*>(acc + CELLS);
    float* const inverse = rad + DIRECT_NODES;
    uint32_t* const box = reinterpret_cast<uint32_t*>(inverse + DIRECT_NODES);
    int* const item0 = reinterpret_cast<int*>(box + DIRECT_NODES);
    int* const node0 = item0 + CELLS;
    if (threadIdx.x < DIRECT_NODES) {
        const int q = threadIdx.x;
        // this quadrature node: panel q / 8, node q % 8 (mirror pairs)
        const int panel = q / 8, k = q % 8;
        const double gx = k < 4 ? -c_gl_x[3 - k] : c_gl_x[k - 4];
        const double gw = k < 4 ? c_gl_w[3 - k] : c_gl_w[k - 4];
        const double n1 = A.n1, n2 = A.n2;
        const double th_max = n2 < n1 ? asin(n2 / n1) : 0.5 * 3.141592653589793;
        const double t0 = th_max * panel / 8.0, t1 = th_max * (panel + 1) / 8.0;
        const double th = t0 + 0.5 * (t1 - t0) * (gx + 1.0);
        const double c = cos(th), sn = sin(th);
        // Fresnel transmission at the readout face (as fresnel_R, in Float64)
        double T = 0.0;
        const double q2 = (n1 / n2) * (n1 / n2);
        const double sin2t = q2 * (1.0 - c * c);
        if (sin2t < 1.0) {
            const double ct = sqrt(1.0 - sin2t);
            const double a = (n1 * c - n2 * ct) / (n1 * c + n2 * ct);
            const double b = (n1 * ct - n2 * c) / (n1 * ct + n2 * c);
            T = 1.0 - 0.5 * (a * a + b * b);
        }
        s_w[q] = 0.5 * (t1 - t0) * gw * T * sn / (4.0 * 3.141592653589793);
        s_c[q] = c;
        s_tan[q] = (float)(sn / c);
    }
    __syncthreads();
    auto x_edge = [&](int e) { return e == nx ? A.L0 : fminf(e * A.pitch, A.L0); };
    auto y_edge = [&](int e) { return e == ny ? A.L1 : fminf(e * A.pitch, A.L1); };
    const int64_t stride = (int64_t)gridDim.x * DIRECT_WARPS;
    for (int64_t i = (int64_t)blockIdx.x * DIRECT_WARPS + (threadIdx.x >> 5); i < A.n; i += stride) {
        const int64_t at = A.site ? A.site[i] : i;
        const float x0 = A.xyz[3 * at], y0 = A.xyz[3 * at + 1], z0 = A.xyz[3 * at + 2];
        const float h = A.L2 - z0;
        const bool inside = h > 0.0f && x0 >= 0.0f && x0 <= A.L0 && y0 >= 0.0f && y0 <= A.L1;   // warp-uniform
        if (inside) {
            // ---- the crossing angles of this lane's two nodes ----
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                const int q = lane + 32 * m;
                const float rho = h * s_tan[q];
                const float inv = 1.0f / rho;
                int ilo = (int)floorf((x0 - rho) / A.pitch), ihi = (int)floorf((x0 + rho) / A.pitch);
                int jlo = (int)floorf((y0 - rho) / A.pitch), jhi = (int)floorf((y0 + rho) / A.pitch);
                // the last column and row reach the face edge, beyond nx and ny pitches too
                ilo = max(ilo, 0); jlo = max(jlo, 0); ihi = min(ihi, nx - 1); jhi = min(jhi, ny - 1);
                ilo = min(ilo, ihi); jlo = min(jlo, jhi);
                if (XTAB)
                    for (int e = ilo; e <= ihi + 1; ++e)
                        aa[e * DIRECT_STRIDE + q] = column_angle((x_edge(e) - x0) * inv);
                if (YTAB)
                    for (int e = jlo; e <= jhi + 1; ++e)
                        ba[e * DIRECT_STRIDE + q] = row_angle((y_edge(e) - y0) * inv);
                wt[q] = (double)(float)(s_w[q] * exp(-(double)A.mu * (double)h / s_c[q])) * DIRECT_FIX;
                rad[q] = rho;
                inverse[q] = inv;
                box[q] = (uint32_t)ilo | (uint32_t)ihi << 8 | (uint32_t)jlo << 16 | (uint32_t)jhi << 24;
            }
        }
        __syncwarp();
        // ---- the nodes whose circle crosses each pixel: [first, first + count),
        // from the one that reaches the pixel (and whose bounding box does) to the
        // last within its farthest corner; two pixels per lane ----
        int total = 0;
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const int c = lane + 32 * m, jj = c / nx, ii = c - jj * nx;
            int first = 0, end = 0;
            if (inside) {
                const float xa = ii * A.pitch - x0, xb = (ii == nx - 1 ? A.L0 : (ii + 1) * A.pitch) - x0;
                const float ya = jj * A.pitch - y0, yb = (jj == ny - 1 ? A.L1 : (jj + 1) * A.pitch) - y0;
                const float nx_ = fmaxf(fmaxf(xa, -xb), 0.0f), ny_ = fmaxf(fmaxf(ya, -yb), 0.0f);
                const float fx = fmaxf(fabsf(xa), fabsf(xb)), fy = fmaxf(fabsf(ya), fabsf(yb));
                const float near2 = (nx_ * nx_ + ny_ * ny_) * 0.999f, far2 = (fx * fx + fy * fy) * 1.001f;
                auto reached = [&](int q) {
                    const uint32_t g = box[q];
                    return rad[q] * rad[q] >= near2 && ii >= (int)(g & 255u) && ii <= (int)((g >> 8) & 255u) &&
                           jj >= (int)((g >> 16) & 255u) && jj <= (int)(g >> 24);
                };
                for (int step = DIRECT_NODES / 2; step > 0; step >>= 1) {
                    if (!reached(first + step - 1)) first += step;
                    if (rad[end + step - 1] * rad[end + step - 1] <= far2) end += step;
                }
                if (!reached(first)) first = DIRECT_NODES;
                if (end == DIRECT_NODES - 1 && rad[end] * rad[end] <= far2) end = DIRECT_NODES;
            }
            const int count = max(end - first, 0);
            // items before this pixel's (pixel order)
            int before = count;
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, before, o);
                if (lane >= o) before += up;
            }
            item0[c] = total + before - count;
            node0[c] = first;
            total += __shfl_sync(0xffffffffu, before, 31);
            acc[c] = 0ull;
        }
        __syncwarp();
        // ---- the (pixel, node) items, an equal run of them per lane ----
        const int per = (total + 31) >> 5;
        int item = lane * per;
        const int last = min(item + per, total);
        if (item < last) {
            int c = 0;                                // the pixel of the first item: the last one starting at or before it
            for (int step = CELLS / 2; step > 0; step >>= 1)
                if (item0[c + step] <= item) c += step;
            while (item < last) {
                const int next = c + 1 < CELLS ? item0[c + 1] : total;
                const int jj = c / nx, ii = c - jj * nx;
                int q = node0[c] + item - item0[c];
                const float* pa = aa + ii * DIRECT_STRIDE;
                const float* pb = ba + jj * DIRECT_STRIDE;
                const float xa = x_edge(ii) - x0, xb = x_edge(ii + 1) - x0;      // where not tabulated
                const float ya = y_edge(jj) - y0, yb = y_edge(jj + 1) - y0;
                unsigned long long sum = 0ull;
                for (const int stop = min(next, last); item < stop; ++item, ++q) {
                    // azimuths with cos(phi) between the columns' edges: x1 in
                    // [0, pi], x2 in [pi, 2 pi]
                    const float a0 = XTAB ? pa[q] : column_angle(xa * inverse[q]);
                    const float a1 = XTAB ? pa[q + DIRECT_STRIDE] : column_angle(xb * inverse[q]);      // a1 <= a0
                    const float x1l = a1, x1h = a0, x2l = TWO_PI_ARC - a0, x2h = TWO_PI_ARC - a1;
                    // and sin(phi) between the rows': y1 where it is positive on
                    // [0, pi/2], y2 around pi, y3 where it is negative on [3 pi/2, 2 pi]
                    const float b0 = YTAB ? pb[q] : row_angle(ya * inverse[q]);         // in [-pi/2, pi/2]
                    const float b1 = YTAB ? pb[q + DIRECT_STRIDE] : row_angle(yb * inverse[q]);
                    const float pi = 0.5f * TWO_PI_ARC;
                    const float y1l = fmaxf(b0, 0.0f), y1h = fmaxf(b1, 0.0f);
                    const float y2l = pi - b1, y2h = pi - b0;
                    const float y3l = b0 + TWO_PI_ARC, y3h = fminf(b1, 0.0f) + TWO_PI_ARC;
                    // x1 never meets y3, nor x2 y1
                    float arc = fmaxf(0.0f, fminf(x1h, y1h) - fmaxf(x1l, y1l));
                    arc += fmaxf(0.0f, fminf(x1h, y2h) - fmaxf(x1l, y2l));
                    arc += fmaxf(0.0f, fminf(x2h, y3h) - fmaxf(x2l, y3l));
                    arc += fmaxf(0.0f, fminf(x2h, y2h) - fmaxf(x2l, y2l));
                    // wt * arc rounded to an integer: the low bits of the sum with 1.5 2^52
                    sum += (unsigned long long)__double_as_longlong(fma(wt[q], (double)arc, 0x1.8p52)) -
                           0x4338000000000000ull;
                }
                if (sum) atomicAdd(&acc[c], sum);
                ++c;
            }
        }
        __syncwarp();
#pragma unroll
        for (int m = 0; m < 2; ++m) A.out[i * CELLS + lane + 32 * m] = (float)((double)acc[lane + 32 * m] / DIRECT_FIX);
        __syncwarp();
    }
}

// Network inputs of the sites: x, y scaled to [-1, 1] and the depth through
// w(t) = (1 - a) t + a (1 - sqrt(1 - t)), t = (z - z0) / Lz clamped to [0, 1].
__global__ void surrogate_inputs(const float* __restrict__ xyz, const int32_t* __restrict__ site, int64_t n, float L0,
                                 float L1, float L2, float z0, float a, float* __restrict__ out)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t at = site ? site[i] : i;
        const float x = xyz[3 * at], y = xyz[3 * at + 1], z = xyz[3 * at + 2] - z0;
        const float t = fminf(fmaxf(z / L2, 0.0f), 1.0f);
        const float w = (1.0f - a) * t + a * (1.0f - sqrtf(1.0f - t));
        out[3 * i] = 2.0f * x / L0 - 1.0f;
        out[3 * i + 1] = 2.0f * y / L1 - 1.0f;
        out[3 * i + 2] = 2.0f * w - 1.0f;
    }
}

// Which ensemble serves each site: the last expert whose depth range holds it,
// else the main one (group 0; expert e is group e + 1).  Each group's sites are
// listed in list + group * n, count[group] of them, 32 consecutive sites at a
// time.  Evaluating the main ensemble everywhere and then the experts over it
// cost the experts' sites twice: every network, the first-pass term and five
// copies (42,001 sites, a third of them an expert's: 781 us, 549 so).
constexpr int SITE_GROUPS = 257;
struct SplitArgs {
    const float* xyz;
    int64_t n;
    int32_t experts;
    float lo[SITE_GROUPS - 1], hi[SITE_GROUPS - 1];
    int32_t* list;
    int32_t* count;
};
__global__ void __launch_bounds__(256) surrogate_split(const __grid_constant__ SplitArgs A)
{
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t w = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); 32 * w < A.n; w += warps) {
        const int64_t i = 32 * w + lane;
        int group = -1;
        if (i < A.n) {
            const float z = A.xyz[3 * i + 2];
            group = 0;
            for (int e = 0; e < A.experts; ++e)
                if (z >= A.lo[e] && z <= A.hi[e]) group = e + 1;
        }
        unsigned left = __ballot_sync(0xffffffffu, group >= 0);
        while (left) {                               // one group of the warp's sites after another
            const int g = __shfl_sync(0xffffffffu, group, __ffs(left) - 1);
            const unsigned same = __ballot_sync(0xffffffffu, group == g);
            int at = 0;
            if (lane == __ffs(same) - 1) at = atomicAdd(A.count + g, __popc(same));
            at = __shfl_sync(0xffffffffu, at, __ffs(same) - 1) + __popc(same & ((1u << lane) - 1u));
            if (group == g) A.list[(int64_t)g * A.n + at] = (int32_t)i;
            left &= ~same;
        }
    }
}

// Diagnostics: fn 0 = binomial(n = par[0], p = par[1]) -> int64,
// fn 1 = emg_min(k = par[0], mu = par[1], sigma = par[2], tau = par[3]) -> double.
__global__ void debug_sampler(int fn, double p0, double p1, double p2, double p3, int64_t n,
                              uint32_t k0, uint32_t k1, void* out, unsigned int* err)
{
    unsigned bad = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        Uni U;
        U.init((uint64_t)i, k0, k1);
        if (fn == 0) ((int64_t*)out)[i] = binomial((int64_t)p0, p1, U, bad);
        else ((double*)out)[i] = emg_min((int64_t)p0, p1, p2, p3, U, bad);
    }
    if (bad && err) atomicOr(err, bad);
}

}  // namespace sur

cudaError_t launch_surrogate_sample(const SurSampleArgs& a, int num_sms, cudaStream_t st)
{
    if (a.n <= 0) return cudaSuccess;
    if (a.cells < 1 || a.cells > sur::CELLS) return cudaErrorInvalidValue;
    int sites = 1;
    while (sites < 32 && a.n > (int64_t)sites * num_sms * sur::SAMPLE_CTAS * sur::SAMPLE_WARPS) sites *= 2;
    const int64_t want = (a.n + sites * sur::SAMPLE_WARPS - 1) / (sites * sur::SAMPLE_WARPS);
    const int64_t cap = (int64_t)num_sms * 16;
    sur::surrogate_sample<<<(unsigned)(want < cap ? want : cap), 32 * sur::SAMPLE_WARPS, 0, st>>>(a, sites);
    return cudaGetLastError();
}

}  // namespace cl

extern "C" {

int cl_surrogate_combine(const float* d_raw, int32_t members, int64_t n_sites,
                         const float* d_y_mean, const float* d_y_std, const float* d_xyz,
                         const cl_box* box, const cl_readout* ro, float pde,
                         float spread_max, float wall_min_mm,
                         float* d_p, float* d_tmean, float* d_tsig, float* d_spread,
                         uint8_t* d_flag, void* stream)
{
    return cl_surrogate_combine_direct(d_raw, members, n_sites, d_y_mean, d_y_std, d_xyz, nullptr, box, ro, pde,
                                       spread_max, wall_min_mm, d_p, d_tmean, d_tsig, d_spread, d_flag, stream);
}

int cl_surrogate_combine_direct(const float* d_raw, int32_t members, int64_t n_sites,
                                const float* d_y_mean, const float* d_y_std, const float* d_xyz,
                                const float* d_direct, const cl_box* box, const cl_readout* ro, float pde,
                                float spread_max, float wall_min_mm,
                                float* d_p, float* d_tmean, float* d_tsig, float* d_spread,
                                uint8_t* d_flag, void* stream)
{
    return cl_surrogate_combine_sites(d_raw, members, n_sites, d_y_mean, d_y_std, d_xyz, nullptr, d_direct, box, ro, pde,
                                      spread_max, wall_min_mm, d_p, d_tmean, d_tsig, d_spread, d_flag, stream);
}

int cl_surrogate_combine_sites(const float* d_raw, int32_t members, int64_t n_sites,
                               const float* d_y_mean, const float* d_y_std, const float* d_xyz,
                               const int32_t* d_site, const float* d_direct, const cl_box* box, const cl_readout* ro,
                               float pde, float spread_max, float wall_min_mm,
                               float* d_p, float* d_tmean, float* d_tsig, float* d_spread,
                               uint8_t* d_flag, void* stream)
{
    if (!box || !ro || members < 1 || n_sites < 0) return CL_ERR_ARG;
    if ((int64_t)ro->grid.nx * ro->grid.ny != cl::sur::CELLS) return CL_ERR_ARG;
    if (n_sites == 0) return CL_OK;
    if (!d_raw || !d_y_mean || !d_y_std || !d_xyz || !d_p || !d_tmean || !d_tsig || !d_spread || !d_flag)
        return CL_ERR_ARG;
    if (!(pde >= 0.0f && pde <= 1.0f)) return CL_ERR_ARG;
    cl::sur::CombineArgs a;
    a.raw = d_raw; a.K = members; a.n = n_sites; a.y_mean = d_y_mean; a.y_std = d_y_std; a.xyz = d_xyz;
    a.site = d_site; a.direct = d_direct;
    a.L0 = box->L[0]; a.L1 = box->L[1]; a.L2 = box->L[2];
    a.front_wrapped = ro->two_sided ? 0 : 1;
    a.pde = pde; a.spread_max = spread_max; a.wall_min_mm = wall_min_mm;
    a.p = d_p; a.tmean = d_tmean; a.tsig = d_tsig; a.spread = d_spread; a.flag = d_flag;
    const int64_t want = (n_sites + cl::sur::COMBINE_WARPS - 1) / cl::sur::COMBINE_WARPS;
    const unsigned grid = (unsigned)(want < 148 * 16 ? want : 148 * 16);
    cl::sur::surrogate_combine<<<grid, 32 * cl::sur::COMBINE_WARPS, 0, (cudaStream_t)stream>>>(a);
    return cudaGetLastError() == cudaSuccess ? CL_OK : CL_ERR_CUDA;
}

int cl_surrogate_direct(const float* d_xyz, int64_t n_sites, const cl_box* box, const cl_optical_params* op,
                        const cl_readout* ro, float* d_out, void* stream)
{
    return cl_surrogate_direct_sites(d_xyz, nullptr, n_sites, box, op, ro, d_out, stream);
}

int cl_surrogate_direct_sites(const float* d_xyz, const int32_t* d_site, int64_t n_sites, const cl_box* box,
                              const cl_optical_params* op, const cl_readout* ro, float* d_out, void* stream)
{
    if (!box || !op || !ro || n_sites < 0) return CL_ERR_ARG;
    if ((int64_t)ro->grid.nx * ro->grid.ny != cl::sur::CELLS || ro->grid.nx < 1 || !(ro->grid.pitch_mm > 0.0f))
        return CL_ERR_ARG;
    // the model: one full readout face at z = Lz
    if (ro->disc || ro->two_sided) return CL_ERR_ARG;
    if (!(op->n_crystal > 0.0f) || !(op->n_coupling > 0.0f) || !(op->abs_len_mm > 0.0f) || !(op->rayleigh_mm > 0.0f))
        return CL_ERR_ARG;
    if (n_sites == 0) return CL_OK;
    if (!d_xyz || !d_out) return CL_ERR_ARG;
    cl::sur::DirectArgs a;
    a.xyz = d_xyz; a.site = d_site; a.n = n_sites; a.L0 = box->L[0]; a.L1 = box->L[1]; a.L2 = box->L[2];
    a.n1 = op->n_crystal; a.n2 = op->n_coupling;
    a.mu = (float)((std::isinf(op->abs_len_mm) ? 0.0 : 1.0 / (double)op->abs_len_mm) +
                   (std::isinf(op->rayleigh_mm) ? 0.0 : 1.0 / (double)op->rayleigh_mm));
    a.pitch = ro->grid.pitch_mm; a.nx = ro->grid.nx; a.ny = ro->grid.ny; a.out = d_out;
    const int64_t want = (n_sites + cl::sur::DIRECT_WARPS - 1) / cl::sur::DIRECT_WARPS;
    const unsigned grid = (unsigned)(want < 148 * 8 ? want : 148 * 8);
    const bool xt = a.nx <= cl::sur::DIRECT_TABULATED, yt = a.ny <= cl::sur::DIRECT_TABULATED;
    const int edges = (xt ? a.nx + 1 : 0) + (yt ? a.ny + 1 : 0);
    const size_t smem = cl::sur::DIRECT_WARPS * cl::sur::direct_warp_floats(edges) * sizeof(float);
    auto kern = !xt ? cl::sur::surrogate_direct<false, true> : !yt ? cl::sur::surrogate_direct<true, false>
                                                                   : cl::sur::surrogate_direct<true, true>;
    // the opt-in is per device and for the most edges tabulated, whatever this
    // grid's are, since threads may launch different grids
    constexpr size_t most = cl::sur::DIRECT_WARPS * cl::sur::direct_warp_floats(cl::sur::DIRECT_MAX_EDGES) * sizeof(float);
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most) != cudaSuccess) {
        cudaGetLastError();
        return CL_ERR_CUDA;
    }
    kern<<<grid, 32 * cl::sur::DIRECT_WARPS, smem, (cudaStream_t)stream>>>(a);
    return cudaGetLastError() == cudaSuccess ? CL_OK : CL_ERR_CUDA;
}

int cl_surrogate_inputs(const float* d_xyz, int64_t n_sites, const cl_box* box, float z_warp, float* d_out,
                        void* stream)
{
    return cl_surrogate_inputs_sites(d_xyz, nullptr, n_sites, box, 0.0f, z_warp, d_out, stream);
}

int cl_surrogate_inputs_sites(const float* d_xyz, const int32_t* d_site, int64_t n_sites, const cl_box* box, float z0,
                              float z_warp, float* d_out, void* stream)
{
    if (!box || n_sites < 0 || !(z_warp >= 0.0f && z_warp <= 1.0f)) return CL_ERR_ARG;
    if (n_sites == 0) return CL_OK;
    if (!d_xyz || !d_out) return CL_ERR_ARG;
    const int64_t want = (n_sites + 255) / 256;
    const unsigned grid = (unsigned)(want < 148 * 32 ? want : 148 * 32);
    cl::sur::surrogate_inputs<<<grid, 256, 0, (cudaStream_t)stream>>>(d_xyz, d_site, n_sites, box->L[0], box->L[1],
                                                                      box->L[2], z0, z_warp, d_out);
    return cudaGetLastError() == cudaSuccess ? CL_OK : CL_ERR_CUDA;
}

int cl_surrogate_split(const float* d_xyz, int64_t n_sites, int32_t experts, const float* lo, const float* hi,
                       int32_t* d_list, int32_t* d_count, int32_t* count, void* stream)
{
    if (n_sites < 0 || n_sites > 0x7fffffff || experts < 0 || experts >= cl::sur::SITE_GROUPS || (experts > 0 && (!lo || !hi)) ||
        !d_list || !d_count || !count || (n_sites > 0 && !d_xyz))
        return CL_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    cl::sur::SplitArgs a;
    a.xyz = d_xyz; a.n = n_sites; a.experts = experts; a.list = d_list; a.count = d_count;
    for (int e = 0; e < experts; ++e) { a.lo[e] = lo[e]; a.hi[e] = hi[e]; }
    const size_t bytes = (size_t)(experts + 1) * sizeof(int32_t);
    if (cudaMemsetAsync(d_count, 0, bytes, st) != cudaSuccess) return CL_ERR_CUDA;
    const int64_t want = (n_sites + 255) / 256;
    if (want > 0) cl::sur::surrogate_split<<<(unsigned)(want < 148 * 8 ? want : 148 * 8), 256, 0, st>>>(a);
    if (cudaGetLastError() != cudaSuccess || cudaMemcpyAsync(count, d_count, bytes, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return CL_ERR_CUDA;
    return CL_OK;
}

int cl_debug_sampler(int fn, const double* par, int64_t n, uint64_t seed, void* d_out,
                     unsigned int* d_err, void* stream)
{
    if ((fn != 0 && fn != 1) || !par || n < 0 || (n > 0 && !d_out)) return CL_ERR_ARG;
    if (n == 0) return CL_OK;
    const unsigned grid = (unsigned)((n + 255) / 256 < 148 * 16 ? (n + 255) / 256 : 148 * 16);
    cl::sur::debug_sampler<<<grid, 256, 0, (cudaStream_t)stream>>>(fn, par[0], par[1], par[2], par[3], n,
                                                                   (uint32_t)seed, (uint32_t)(seed >> 32),
                                                                   d_out, d_err);
    return cudaGetLastError() == cudaSuccess ? CL_OK : CL_ERR_CUDA;
}

}  // extern "C"
