// cl_transport.cu — sm_100a transport kernels and the C-ABI of
// include/crysplight_cuda.h.
//
// Kernel design (B200):
//   * persistent grid: (#SM x resident CTAs) CTAs of 256 threads; every warp
//     claims photon chunks from a device work queue (one 64-bit atomic per
//     chunk) and each lane refills itself with the next photon the moment
//     its photon terminates, so long-bouncing photons never idle a warp;
//   * parameters travel as a __grid_constant__ kernel argument (constant
//     bank), the sincos and log reduction tables sit in shared memory;
//   * point mode: where they fit, the nx*ny*(nbins+1) count tile and the nx*ny
//     first-time tile live in shared memory; one atomic add per detection,
//     first times by atomicMin on order-preserving uint32 keys where the
//     photon is earlier than the key; each CTA flushes its tile once with
//     coalesced global atomics and the last CTA decodes the first-time keys in
//     place;
//   * segment mode (scan points, 511 keV events): per-segment 8x8 maps and
//     first-time keys are reduced with global atomics, one of each per
//     detection, or per distinct slot of a warp where many photons share a slot
//     (add_crowded); a finalize kernel decodes keys and sums npe.
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <cmath>
#include <mutex>
#include <new>

#include <cuda_runtime.h>
#include <curand_philox4x32_x.h>

#include "../../include/crysplight_cuda.h"
#include "cl_device.cuh"
#include "cl_launch.h"
#include "cl_surrogate.cuh"

#define CL_VERSION_STRING "crysplight_b200 0.1.0 (sm_100a)"

namespace cl {

constexpr unsigned FULL = 0xffffffffu;
constexpr int GAUSS_OFF = 1 << 24;    // sqrt(-2 log u) after the 2^24 logs
constexpr int N_COUNTERS = 10;        // cl_counters, then the photon-steps
// Photons per slot from which a launch's detections are added slot by slot
// (segment mode; see add_crowded): few cells, and the 64 of a full map.
constexpr int64_t CROWDED_FEW = 1024, CROWDED = 4096;
constexpr size_t CTA_EXTRA_SMEM = 1024 + 8 * N_COUNTERS * 8 + 16;   // reserved and static shared memory of a CTA
constexpr int SCTAB_BYTES = CLM_SC_N * 16;
constexpr int LOGTAB_BYTES = ((CLM_LOG_NTAB * 16 + 127) / 128) * 128 + SCTAB_BYTES;  // both tables

__constant__ double c_logtab[2 * CLM_LOG_NTAB] = { CLM_LOG_TAB_INIT };
__constant__ double c_sctab[2 * CLM_SC_N] = { CLM_SC_TAB_INIT };

// Copy the log and sincos tables into shared memory (the first LOGTAB_BYTES).
__device__ __forceinline__ void load_tables(unsigned char* smem, double2*& tab, double2*& sctab)
{
    sctab = reinterpret_cast<double2*>(smem);
    tab = reinterpret_cast<double2*>(smem + SCTAB_BYTES);
    for (int i = threadIdx.x; i < CLM_SC_N; i += blockDim.x)
        sctab[i] = make_double2(c_sctab[2 * i], c_sctab[2 * i + 1]);
    for (int i = threadIdx.x; i < CLM_LOG_NTAB; i += blockDim.x)
        tab[i] = make_double2(c_logtab[2 * i], c_logtab[2 * i + 1]);
}

struct KArgs {
    Physics P;
    uint64_t pid0;
    int64_t n;
    int32_t npos;
    int32_t warp_chunk;
    int32_t cells;        // nx*ny
    int32_t bins_total;   // nbins+1
    const float* px; const float* py; const float* pz; const float* pt;
    const int64_t* src_off; const int32_t* src_seg; int64_t n_src; int64_t n_seg;
    uint32_t* counts;     // point: cells*bins_total
    uint32_t* keys;       // point: cells; segments: cells*n_seg
    uint32_t* maps;       // segments: cells*n_seg
    unsigned long long* tsum;   // segments with moments: cells*n_seg
    unsigned long long* tsum2;
    unsigned long long* counters;  // 9 x int64, cl_counters order
    uint8_t* r_status; int16_t* r_idx; float* r_t; int32_t* r_bounces;
    unsigned long long* queue;
    unsigned long long* steps;
    unsigned int* done;
    unsigned int* err;
    unsigned long long* status;   // point: the steps and the error word, beside the outputs (or NULL)
    const float* logtab;  // log u and sqrt(-2 log u) of every uniform (logtab_fill), or NULL: compute
    unsigned long long budget_ns;   // device time budget of the launch, 0 = none
};

// Nanoseconds of the GPU's global timer.
__device__ __forceinline__ unsigned long long globaltimer_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ int time_bin0(float t, const Physics& P)
{
    // 1 + unsafe_trunc(t / bin_ns), overflow -> nbins+1 (src/transport.jl:100-101), 0-based
    const float q = t / P.bin_ns;
    if (!(q < (float)P.nbins)) return P.nbins;
    const int b = (int)q;
    return b < 0 ? 0 : b;
}

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    return v;
}

// The position of photon k (src/kernel.jl:171); out of line, it is a 64-bit division.
static __device__ __noinline__ int32_t position_of(int64_t k, int32_t npos) { return (int32_t)((uint64_t)k % (uint64_t)npos); }

// Rare paths of the transport kernel (these, wall_hit, fresnel_R) are functions
// of their own: inlined, they cost the loop registers and instruction-cache
// room.  Scan 98.0 -> 96.7 (wall_hit, fresnel_R) -> 93.5 ms (find_source),
// 3,001 events 20.2 -> 19.9 -> 19.3 ms.
// Galloping search: largest s >= hint with off[s] <= k (off[n_src] = total).
static __device__ __noinline__ int64_t find_source(const int64_t* __restrict__ off, int64_t n_src,
                                               int64_t hint, int64_t k)
{
    int64_t lo = hint, step = 1;
    int64_t hi = hint + 1;
    while (hi < n_src && __ldg(off + hi) <= k) {
        lo = hi;
        step <<= 1;
        hi = lo + step;
    }
    if (hi > n_src) hi = n_src;
    // invariant: off[lo] <= k < off[hi]  (off[n_src] > k)
    while (hi - lo > 1) {
        const int64_t mid = lo + ((hi - lo) >> 1);
        if (__ldg(off + mid) <= k) lo = mid; else hi = mid;
    }
    return lo;
}

// Adds the detections of a warp's active lanes, all lanes of a slot together:
// one reduction per distinct slot.  Where tens of photons share a slot at any
// time, the reductions on one address are the bound (the L2 takes about one per
// clock); elsewhere finding the lanes out costs more than it saves.  4M photons
// of a crystal that most leave on the first step, one 1x1 segment: 2,880 us one
// by one, 900 so; 8x8: 1,860 and 1,700; 512 segments of 1x1: 2,230 and 930, of
// 8x8: 985 and 1,060.  A scan of 200,000 photons per point and 8x8 map (3,125 a
// slot) takes 93.3 ms one by one and 95.2 so; hence the two thresholds.
static __device__ __noinline__ void add_crowded(uint32_t* maps, uint32_t* keys, unsigned long long slot, uint32_t key)
{
    const unsigned same = __match_any_sync(__activemask(), (uint32_t)slot);
    key = __reduce_min_sync(same, key);
    if ((int)(threadIdx.x & 31) == __ffs(same) - 1) {
        atomicAdd(maps + slot, (uint32_t)__popc(same));
        atomicMin(keys + slot, key);
    }
}

// What a kernel instance computes: counts over the cells and time bins of one
// readout plane; a map per segment; that with arrival-time moments; and the two
// segment modes with crowded slots.
enum : int { POINT = 0, SEGMENTS = 1, MOMENTS = 2, SEGMENTS_CROWDED = 3, MOMENTS_CROWDED = 4 };

// Per-lane transport states of the warp loop.  One loop iteration moves each
// active lane one state forward; a whole wall interaction (move, UNIFIED try,
// wrap) completes in one iteration, so an iteration is about one photon-step.
// States from S_INIT on set a new direction from a polar cosine and an azimuth.
enum : int32_t {
    S_IDLE = 0,   // no photon; below 0: minus the fate of a photon not yet booked
    S_MOVE = 1,   // bulk competition + wall interaction (src/transport.jl:127-233)
    S_UNI = 2,    // another UNIFIED try at the same wall (src/optics.jl:54-78)
    S_INIT = 3,   // emission: direction and time (src/kernel.jl:173-180)
    S_RAY = 4,    // Rayleigh rejection sampling + rotation (src/optics.jl:87-112)
    S_LAMB = 5,   // Lambertian re-injection (src/optics.jl:118-138)
};

#ifndef CL_MIN_CTAS_PER_SM
#define CL_MIN_CTAS_PER_SM 4
#endif

// Optical configurations compiled with their flags as constants (the branches
// they rule out vanish from the loop): SPEC_ESR and SPEC_TEFLON are a rough
// (UNIFIED) back-painted wrap, specular or Lambertian, over a full, one-sided
// readout face with finite absorption and Rayleigh lengths -- the BGO+ESR and
// CsI(Tl)+Teflon run files; SPEC_ANY reads every flag from the parameters.
enum : int { SPEC_ANY = 0, SPEC_ESR = 1, SPEC_TEFLON = 2 };

// log u and sqrt(-2 log u) of a uniform u = k 2^-24: from the tables, or (TAB
// false) evaluated in place.
__device__ __forceinline__ int uniform_index(float u) { return (int)(u * 16777216.0f) - 1; }
template <bool TAB>
__device__ __forceinline__ float uniform_log(const float* __restrict__ tab, float u, const double2* __restrict__ logtab)
{
    return TAB ? __ldg(tab + uniform_index(u)) : cl_logf_u(u, logtab);
}

// The loop computes what decides a photon's next step exactly and everything
// else it can do without: the bound is instruction issue (the state machine's
// selects, moves and branches, not the arithmetic), so
//   * the wall axis comes from approximate reciprocals and only the winning
//     axis is divided; the bulk competition compares the uniforms with
//     approximate survival probabilities; Fresnel compares its uniform with an
//     approximate coefficient.  Each has an error bound, and a lane inside it
//     (about 1e-5 of them; a bulk event always) takes the exact expressions,
//     so every result has the reference's bits;
//   * a lane's next uniforms are read at fixed offsets from one address (the
//     ring is mirrored past its end), and the number consumed is added once;
//   * outcomes are merged by selects into one flip / one new direction / one
//     state change, not one branch each;
//   * the tilt's sqrt(-2 log u) is looked up whole.
//   * booking an ended photon and starting the next one wait for a few free lanes.
// Against the same states with exact expressions and a branch per outcome
// (31.2 -> 20.4 warp instructions per photon-step): BGO+ESR scan of 51.2M
// photons 143.9 -> 100.4 ms (49 G photon-steps/s; 93.5 ms and 18.7 instructions with
// the rare paths out of line), 3,001 CsI(Tl)+Teflon events
// 32.6 -> 20.6 ms (19.3), 10^6-photon CsI(Tl) point 1.17 -> 0.79 ms.
template <int MODE, bool REC, bool TILE, int SPEC, bool TAB>
__global__ void __launch_bounds__(256, CL_MIN_CTAS_PER_SM) transport_kernel(const __grid_constant__ KArgs A)
{
    extern __shared__ __align__(16) unsigned char smem[];
    double2 *s_tab, *s_sctab;
    load_tables(smem, s_tab, s_sctab);
    unsigned char* const s_ring = smem + LOGTAB_BYTES;
    uint32_t* s_counts = reinterpret_cast<uint32_t*>(s_ring + RING_BYTES);
    uint32_t* s_keys = s_counts + (TILE ? A.cells * A.bins_total : 0);
    // per-warp counters (cl_counters order, then the steps); lane i owns entry i
    __shared__ unsigned long long s_cnt[8][N_COUNTERS];
    __shared__ unsigned int s_last;

    const Physics& P = A.P;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    if (TILE) {
        const int nt = A.cells * A.bins_total;
        for (int i = tid; i < nt; i += blockDim.x) s_counts[i] = 0u;
        for (int i = tid; i < A.cells; i += blockDim.x) s_keys[i] = INF_KEY;
    }
    for (int i = tid; i < 8 * N_COUNTERS; i += blockDim.x) (&s_cnt[0][0])[i] = 0ull;
    // every ring word holds a uniform from the start: lanes without a photon
    // read them too, and their table lookups stay in range
    for (int r = 0; r < RING_ROWS; ++r) *reinterpret_cast<float*>(s_ring + r * RING_ROW + 4 * tid) = 1.0f;
    __syncthreads();

    // free lanes that make a turnover worth its cost: 1 / 3 / 4 lanes took 105.5 /
    // 100.5 / 101.0 ms on the scan (a photon ends every 97 steps); 1 / 4 / 8 / 10
    // lanes 23.8 / 21.3 / 20.5 / 20.6 ms on the events (every 12 steps).  The
    // general instance serves short and long lives: 3 / 5 / 8 lanes take 1,230 /
    // 1,170 / 1,157 us for 2M photons of 14 steps (specular paint), 1,032 / 971 /
    // 959 of 7 (diffuse paint), 6.75 / 6.66 / 7.02 ms of 122 (polished, specular)
    constexpr int TURNOVER = SPEC == SPEC_ESR ? 3 : 8;

    uint32_t* tile_counts = TILE ? s_counts : A.counts;
    uint32_t* tile_keys = TILE ? s_keys : A.keys;
    unsigned long long* my_cnt = s_cnt[tid >> 5];

    const unsigned lt_mask = (1u << lane) - 1u;
    const uint32_t sc0 = smem_addr(smem), ring0 = sc0 + LOGTAB_BYTES;
    const bool air_gap = SPEC != SPEC_ANY || P.air_gap;
    const bool uni_possible = SPEC != SPEC_ANY || (P.air_gap && P.sigma_alpha > 0.0f);
    const bool wrap_specular = SPEC == SPEC_ESR || (SPEC == SPEC_ANY && P.wrap_specular);
    const bool abs_finite = SPEC != SPEC_ANY || P.abs_finite;
    const bool ray_finite = SPEC != SPEC_ANY || P.ray_finite;
    const bool disc = SPEC == SPEC_ANY && P.disc;
    const bool two_sided = SPEC == SPEC_ANY && P.two_sided;
    // states a configuration never reaches (tests on them compile away)
    constexpr bool lamb_possible = SPEC != SPEC_ESR;      // Lambertian wrap or surround
    const float inf = __int_as_float(0x7f800000);
    // uniforms a move draws for the bulk competition, as a byte offset in the ring
    const uint32_t bulk_off = (abs_finite ? RING_ROW : 0) + (ray_finite ? RING_ROW : 0);

    // per-lane photon state
    float x = 0.f, y = 0.f, z = 0.f, ux = 0.f, uy = 0.f, uz = 0.f, t = 0.f;
    int32_t bounces = 0, nscat = 0, st = S_IDLE, face = 1, tries = 0;
    Rng rng;
    rng_init(rng, 0);
    rng_park(rng);
    int32_t seg = 0;
    // warp-uniform work pool
    int64_t pool_lo = 0, pool_hi = 0, pool_src = 0;
    bool exhausted = false;
    bool overrun = false, under = false, timed_out = false;
    // time budget: a warp-uniform iteration count, the clock read every 256
    uint32_t iter = 0;
    const unsigned long long t_begin = A.budget_ns ? globaltimer_ns() : 0ull;

    for (;;) {
        // ---- turnover: book the ended photons, refill their lanes from the
        // warp's pool / the global queue.  Both cost the same for one lane as
        // for many, so lanes wait until TURNOVER of them are free.
        if (__popc(__ballot_sync(FULL, st <= 0)) >= TURNOVER) {
            const unsigned tmask = __ballot_sync(FULL, st < 0);
            if (tmask != 0u) {
                const int32_t status = st < 0 ? -st : ST_FLYING;
                const bool det = status == ST_DETECTED;
                int32_t idx = 0;
                if (det) {
                    // the conversion saturates: inside the grid whatever the pitch
                    const int32_t ii = min((int32_t)(x / P.pitch), P.nx - 1);
                    const int32_t jj = min((int32_t)(y / P.pitch), P.ny - 1);
                    const int32_t cell = jj * P.nx + ii, lin = cell + 1;
                    idx = two_sided && face == FACE_FRONT ? -lin : lin;
                    const uint32_t key = float_key(t);
                    // one reduction per photon: a warp seldom detects two photons in
                    // the same slot, and finding out costs more than it saves
                    if (MODE == POINT) {
                        const int bin = time_bin0(t, P);       // a histogram in global memory may pass 2^31 counts
                        atomicAdd(tile_counts + cell + (TILE ? A.cells * bin : (int64_t)A.cells * bin), 1u);
                        // the cells' keys are hot; most photons are later than the
                        // key already there (which only ever falls)
                        if (key < (TILE ? tile_keys[cell] : __ldcg(tile_keys + cell))) atomicMin(tile_keys + cell, key);
                    } else {
                        // a segment id outside the maps (untrusted device input) drops the detection
                        if (seg >= 0 && (int64_t)seg < A.n_seg) {
                            const unsigned long long slot =
                                (unsigned long long)seg * (unsigned long long)A.cells + (unsigned long long)cell;
                            if (MODE >= SEGMENTS_CROWDED) {
                                add_crowded(A.maps, A.keys, slot, key);
                            } else {
                                atomicAdd(A.maps + slot, 1u);
                                atomicMin(A.keys + slot, key);
                            }
                            if (MODE == MOMENTS || MODE == MOMENTS_CROWDED) {
                                // fixed-point time moments (exact integer sums, order-independent)
                                const float tc = fminf(fmaxf(t, 0.0f), CL_MOMENT_T_MAX_NS);
                                atomicAdd(A.tsum + slot, __float2ull_rn(tc * CL_MOMENT_T_SCALE));
                                atomicAdd(A.tsum2 + slot, __float2ull_rn((tc * tc) * CL_MOMENT_T2_SCALE));
                            }
                        } else {
                            atomicOr(A.err, 16u);
                        }
                    }
                }
                if (REC && st < 0) {
                    const uint64_t k = (((uint64_t)rng.pid_hi << 32) | rng.pid_lo) - A.pid0 - 1ull;
                    if (A.r_status) A.r_status[k] = (uint8_t)status;
                    if (A.r_idx) A.r_idx[k] = (int16_t)idx;
                    if (A.r_t) A.r_t[k] = t;
                    if (A.r_bounces) A.r_bounces[k] = bounces;
                }
                // counters: the fates in five 6-bit fields of one reduction (the
                // caps are what is left of the ended lanes), the sums one each;
                // lane i adds entry i of the warp's own counters
                const uint32_t field = st >= 0 || status == ST_CAP ? 0u
                                       : (1u << (status == ST_DETECTED ? 0 : (status == ST_ABS_SUR ? 24 : 6 * (status - 1))));
                const uint32_t fates = __reduce_add_sync(FULL, field);
                const uint32_t front = two_sided ? (uint32_t)__popc(__ballot_sync(FULL, det && idx < 0)) : 0u;
                const uint32_t sb = __reduce_add_sync(FULL, det ? (uint32_t)bounces : 0u);
                const uint32_t sc = __reduce_add_sync(FULL, st < 0 ? (uint32_t)nscat : 0u);
                const uint32_t ss = __reduce_add_sync(FULL, st < 0 ? (uint32_t)(bounces + (status != ST_CAP)) : 0u);
                if (lane < N_COUNTERS) {
                    // ndet, ndet_front, bulk, wall, sipm, cap, sur, nscat, sum_bounces_det, steps
                    uint32_t add = fates & 63u;
                    if (lane == 1) add = front;
                    if (lane >= 2 && lane <= 4) add = (fates >> (6 * (lane - 1))) & 63u;
                    if (lane == 5) add = (uint32_t)__popc(tmask) - (fates & 63u) - ((fates >> 6) & 63u) -
                                         ((fates >> 12) & 63u) - ((fates >> 18) & 63u) - (fates >> 24);
                    if (lane == 6) add = fates >> 24;
                    if (lane == 7) add = sc;
                    if (lane == 8) add = sb;
                    if (lane == 9) add = ss;
                    my_cnt[lane] += (unsigned long long)add;
                }
                if (st < 0) {
                    st = S_IDLE;
                    rng_park(rng);
                }
            }
            if (!exhausted) {
                const unsigned need = __ballot_sync(FULL, st == S_IDLE);
                const int nneed = __popc(need);
                const int rank = __popc(need & lt_mask);
                int64_t my_k = -1;
                int64_t my_hint = pool_src;
                const int64_t avail = pool_hi - pool_lo;
                const int64_t taken = avail < nneed ? avail : (int64_t)nneed;
                if (st == S_IDLE && rank < taken) my_k = pool_lo + rank;
                pool_lo += taken;
                if (taken < nneed) {
                    unsigned long long base = 0;
                    if (lane == 0) base = atomicAdd(A.queue, (unsigned long long)A.warp_chunk);
                    base = __shfl_sync(FULL, base, 0);
                    if ((int64_t)base >= A.n) {
                        exhausted = true;
                    } else {
                        pool_lo = (int64_t)base;
                        pool_hi = pool_lo + A.warp_chunk;
                        if (pool_hi > A.n) pool_hi = A.n;
                        if (MODE != POINT) {
                            int64_t s0 = 0;
                            if (lane == 0) s0 = find_source(A.src_off, A.n_src, pool_src, pool_lo);
                            pool_src = __shfl_sync(FULL, s0, 0);
                        }
                        const int64_t rem = nneed - taken;
                        const int64_t avail2 = pool_hi - pool_lo;
                        const int64_t taken2 = avail2 < rem ? avail2 : rem;
                        if (st == S_IDLE && rank >= taken && rank - taken < taken2) {
                            my_k = pool_lo + (rank - taken);
                            my_hint = pool_src;
                        }
                        pool_lo += taken2;
                    }
                }
                if (my_k >= 0) {
                    if (MODE == POINT) {
                        const int32_t j = A.npos == 1 ? 0 : position_of(my_k, A.npos);
                        x = __ldg(A.px + j); y = __ldg(A.py + j); z = __ldg(A.pz + j);
                        t = A.pt ? __ldg(A.pt + j) : 0.0f;
                    } else {
                        const int64_t s = find_source(A.src_off, A.n_src, my_hint, my_k);
                        x = __ldg(A.px + s); y = __ldg(A.py + s); z = __ldg(A.pz + s);
                        t = A.pt ? __ldg(A.pt + s) : 0.0f;
                        seg = __ldg(A.src_seg + s);
                    }
                    rng_init(rng, A.pid0 + (uint64_t)my_k + 1ull);
                    bounces = 0; nscat = 0; tries = 0;
                    st = S_INIT;
                }
            }
            if (!__any_sync(FULL, st > 0)) break;
        }
        if (((++iter) & 255u) == 0u && A.budget_ns != 0ull) {
            // photons still in flight are dropped; the host reports CL_ERR_TIMEOUT
            if (__any_sync(FULL, globaltimer_ns() - t_begin > A.budget_ns)) { timed_out = true; break; }
        }

        // ---- top up the uniform ring: one Philox call site for the warp ----
        if (__any_sync(FULL, rng_short(rng))) {
            // every lane with room tops up at this convergent point, so later
            // iterations need the fill less often
            under |= rng_under(rng);
            if (rng_room(rng)) rng_fill(rng, ring0, P.rk);
        }

        // ---- draws: this iteration's uniforms at fixed offsets ----
        const uint32_t w = ring0 + (rng.pos & RING_MASK);
        // the table lookup (tilt's gaussian, or the emission time's log) and the azimuth
        const uint32_t og = st == S_MOVE ? bulk_off : (st == S_INIT ? 2u * RING_ROW : 0u);
        uint32_t oaz = st <= S_UNI ? og + 2u * RING_ROW : RING_ROW;
        float mu = 0.0f;
        bool ray_ok = true;
        if (st == S_RAY) {
            // two rejection tries in one iteration (8 of 9 scatters end in it)
            mu = 1.0f - 2.0f * ring_word(w);
            ray_ok = 2.0f * ring_word(w + RING_ROW) <= 1.0f + mu * mu;
            oaz = 2u * RING_ROW;
            if (!ray_ok) {
                ++tries;
                mu = 1.0f - 2.0f * ring_word(w + 2u * RING_ROW);
                ray_ok = 2.0f * ring_word(w + 3u * RING_ROW) <= 1.0f + mu * mu;
                oaz = 4u * RING_ROW;
            }
        }

        // ---- elementary functions, once per warp (Float64, rounded once) ----
        // Straight-line and unconditional (a lane that needs none of them reads
        // some other uniform), so that their latencies overlap.
        const uint32_t v = w + og;
        const float ug = ring_word(v);
        float G;                    // sqrt(-2 log u); for an emission the log itself
        if (TAB) {
            G = __ldg(A.logtab + uniform_index(ug) + (st == S_INIT ? 0 : GAUSS_OFF));
        } else {
            G = cl_logf_u(ug, s_tab);
            if (st != S_INIT) G = sqrtf(-2.0f * G);
        }
        float s0, c0, s1, c1;
        cl_sincosf_core(TWO_PI_F * ring_word(v + RING_ROW), sc0, &s0, &c0);
        cl_sincosf_core(TWO_PI_F * ring_word(w + oaz), sc0, &s1, &c1);

        bool done = false;          // an interaction that counts as a bounce
        if (st >= S_INIT) {
            // ---- a new direction: emission, Rayleigh scatter, Lambertian lobe ----
            float c = mu;
            if (st != S_RAY) {
                const float u = ring_word(w);
                c = lamb_possible && st == S_LAMB ? sqrt_mid(u) : 1.0f - 2.0f * u;
            }
            const float sn = sqrt_mid(fmaxf(0.0f, 1.0f - c * c));
            const float a = sn * c1, b = sn * s1;
            rng.pos += oaz + (ray_ok ? RING_ROW : 0u);
            if (st == S_RAY) {
                if (ray_ok || ++tries >= 4096) {
                    overrun |= !ray_ok;
                    rayleigh_rotate(c, a, b, ux, uy, uz);
                    nscat += 1;
                    done = true;
                }
            } else if (lamb_possible && st == S_LAMB) {
                lambertian_from(face, c, a, b, ux, uy, uz);
                done = true;
            } else {
                ux = a; uy = b; uz = c;
                if (P.tau > 0.0f) { t += (-P.tau) * G; rng.pos += RING_ROW; }
                st = S_MOVE;
            }
        } else if (st > 0) {
            // ---- the step to the wall; another try (S_UNI) is a step of length 0
            // at the wall it is on ----
            float d, cosw;          // distance and |cos| of the incidence on the wall
            int32_t f;
            if (!wall_hit_fast(P, x, y, z, ux, uy, uz, d, f, cosw) && st == S_MOVE) {
                f = wall_hit(P, x, y, z, ux, uy, uz, d);
                cosw = fabsf(f <= 2 ? ux : (f <= 4 ? uy : uz));
            }
            if (st != S_MOVE) { d = 0.0f; f = face; }
            else { tries = 0; face = f; }
            const float u_abs = ring_word(w);
            const float u_ray = ring_word(w + (abs_finite ? RING_ROW : 0u));
            bool hit = true;
            rng.pos += og;
            // no bulk interaction if each uniform is clearly below its
            // survival probability exp(-d / length): the path length
            // -length log u is then clearly above d.  (Another try moves by 0, below
            // which no path length is but one of a negative length, SPEC_ANY's.)
            if ((SPEC != SPEC_ANY || st == S_MOVE) &&
                !((!abs_finite || u_abs < survive_below(d, P.abs_rate)) &&
                  (!ray_finite || u_ray < survive_below(d, P.ray_rate)))) {
                const float d_abs = abs_finite ? (-P.abs_len) * uniform_log<TAB>(A.logtab, u_abs, s_tab) : inf;
                const float d_ray = ray_finite ? (-P.ray_len) * uniform_log<TAB>(A.logtab, u_ray, s_tab) : inf;
                if (d_abs < d && d_abs <= d_ray) {
                    st = -ST_ABS_BULK;
                    hit = false;
                } else if (d_ray < d) {
                    x += d_ray * ux; y += d_ray * uy; z += d_ray * uz;
                    t += d_ray * P.inv_v;
                    st = S_RAY;
                    hit = false;
                }
            }
            if (hit) {
                // advance to the wall: clamp, then snap the hit axis (src/transport.jl:146-157)
                const bool on_x = f <= 2, on_y = !on_x && f <= 4, on_z = f > 4, outer = (f & 1) != 0;
                const float nx_ = x + d * ux, ny_ = y + d * uy, nz_ = z + d * uz;
                x = on_x ? (outer ? P.L0 : 0.0f) : clamp_to(nx_, P.L0);
                y = on_y ? (outer ? P.L1 : 0.0f) : clamp_to(ny_, P.L1);
                z = on_z ? (outer ? P.L2 : 0.0f) : clamp_to(nz_, P.L2);
                t += d * P.inv_v;
                // ---- the wall interaction; uniforms from v on ----
                const float sgn = outer ? 1.0f : -1.0f;      // outward normal component
                const bool readout = f == FACE_BACK || (two_sided && f == FACE_FRONT);
                bool flip = false, take = false;
                float rx = 0.f, ry = 0.f, rz = 0.f;
                if (SPEC == SPEC_ANY && !readout && !air_gap) {
                    // front-painted wrap, src/transport.jl:186-198
                    rng.pos += RING_ROW;
                    if (ug <= P.wrap_R) {
                        if (wrap_specular) flip = true;
                        else st = S_LAMB;
                    } else {
                        st = -ST_ABS_WALL;
                    }
                } else {
                    // UNIFIED facet (src/optics.jl:55-66); a readout lane computes
                    // one too and does not use it
                    const bool facet = uni_possible && !readout;
                    bool retry = false;
                    float Nfx = 0.f, Nfy = 0.f, Nfz = 0.f, fcos = cosw;
                    uint32_t fo = 0;             // offset of the Fresnel uniform
                    if (uni_possible) {
                        const float alpha = P.sigma_alpha * fabsf(G * c0);
                        float sa, ca;
                        cl_sincosf_core(fminf(alpha, 1.2f), sc0, &sa, &ca);
                        const float b = sa * c1, c = sa * s1, n = ca * sgn;
                        Nfx = on_x ? n : b;
                        Nfy = on_y ? n : (on_x ? b : c);
                        Nfz = on_z ? n : c;
                        const float cosi = ux * Nfx + uy * Nfy + uz * Nfz;
                        if (facet) {
                            fcos = cosi;
                            // a tilt out of range is drawn again before its azimuth is
                            retry = alpha >= 1.2f || cosi <= 0.0f;
                            fo = alpha >= 1.2f ? 2u * RING_ROW : 3u * RING_ROW;
                        }
                    }
                    // Fresnel (src/optics.jl:10-19)
                    const float sin2t = (readout ? P.qc2 : P.qa2) * (1.0f - fcos * fcos);
                    const float uf = ring_word(v + fo), un = ring_word(v + fo + RING_ROW);
                    const bool refl = fresnel_reflects(P, readout ? P.n_coupling : 1.0f, sin2t, fcos, uf);
                    rng.pos += fo + (retry || sin2t >= 1.0f ? 0u : (refl ? RING_ROW : 2u * RING_ROW));
                    // facet reflection, kept only if it points back into the
                    // crystal (src/optics.jl:68-77)
                    rx = ux - (2.0f * fcos) * Nfx;
                    ry = uy - (2.0f * fcos) * Nfy;
                    rz = uz - (2.0f * fcos) * Nfz;
                    const bool inward = sgn * (on_x ? rx : (on_y ? ry : rz)) < 0.0f;
                    take = facet && refl && !retry && inward;
                    flip = !facet && refl;
                    if (!refl && !retry) {
                        // through the interface: a SiPM or its surround, or the
                        // reflector behind the air gap (src/transport.jl:161-225)
                        const bool sipm = readout && (!disc || (x - P.cx) * (x - P.cx) + (y - P.cy) * (y - P.cy) <= P.r2);
                        const bool kept = un <= (sipm ? P.pde : (SPEC == SPEC_ANY && readout ? P.sur_R : P.wrap_R));
                        if (sipm) {
                            st = kept ? -ST_DETECTED : -ST_ABS_SIPM;
                        } else if (kept) {
                            if (SPEC == SPEC_ANY && readout ? P.sur_specular : wrap_specular) flip = true;
                            else st = S_LAMB;
                        } else {
                            st = SPEC == SPEC_ANY && readout ? -ST_ABS_SUR : -ST_ABS_WALL;
                        }
                    }
                    if (retry || (facet && refl && !inward)) {
                        if (++tries >= 20) flip = true;
                        else st = S_UNI;
                    }
                }
                ux = take ? rx : (flip && on_x ? -ux : ux);
                uy = take ? ry : (flip && on_y ? -uy : uy);
                uz = take ? rz : (flip && on_z ? -uz : uz);
                done = take || flip;
            }
        }

        // end of an interaction: count the bounce (src/transport.jl:228-232)
        if (done) {
            bounces += 1;
            st = bounces >= P.max_bounces ? -ST_CAP : S_MOVE;
        }
    }
    if (overrun) atomicOr(A.err, 1u);
    if (under) atomicOr(A.err, 2u);
    if (timed_out && lane == 0) atomicOr(A.err, 32u);
    __syncthreads();

    // ---- one coalesced flush per CTA ----
    if (TILE) {
        const int nt = A.cells * A.bins_total;
        for (int i = tid; i < nt; i += blockDim.x) {
            const uint32_t v = s_counts[i];
            if (v) atomicAdd(A.counts + i, v);
        }
        for (int i = tid; i < A.cells; i += blockDim.x) {
            const uint32_t kk = s_keys[i];
            if (kk != INF_KEY) atomicMin(A.keys + i, kk);
        }
    }
    if (tid < N_COUNTERS) {
        unsigned long long v = 0;
        for (int q = 0; q < 8; ++q) v += s_cnt[q][tid];
        if (v) atomicAdd(tid < 9 ? A.counters + tid : A.steps, v);
    }

    if (MODE == POINT) {
        // last CTA decodes the first-time keys into Float32 in place
        __threadfence();
        __syncthreads();
        if (tid == 0) s_last = (atomicAdd(A.done, 1u) == gridDim.x - 1u) ? 1u : 0u;
        __syncthreads();
        if (s_last) {
            __threadfence();
            for (int i = tid; i < A.cells; i += blockDim.x) {
                const uint32_t kk = __ldcg(A.keys + i);
                A.keys[i] = __float_as_uint(key_float(kk));
            }
            if (tid == 0 && A.status) {
                A.status[0] = __ldcg(A.steps);
                A.status[1] = __ldcg(A.err);
            }
        }
    }
}

// Zero the outputs and the work queue before a launch.
__global__ void init_kernel(uint32_t* counts, int64_t n_counts, uint32_t* keys, int64_t n_keys,
                            unsigned long long* counters, unsigned long long* queue,
                            unsigned long long* steps, unsigned int* done, unsigned int* err)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (int64_t i = i0; i < n_counts; i += stride) counts[i] = 0u;
    for (int64_t i = i0; i < n_keys; i += stride) keys[i] = INF_KEY;
    if (i0 < 9) counters[i0] = 0ull;
    if (i0 == 0) { *queue = 0ull; *steps = 0ull; *done = 0u; *err = 0u; }
}

// The tables of the uniforms u = (k+1) 2^-24, k < 2^24: t[k] = log u and
// t[GAUSS_OFF + k] = sqrt(-2 log u), the same functions and rounding as the
// computed path.
__global__ void logtab_fill(float* t)
{
    extern __shared__ __align__(16) unsigned char smem[];
    double2 *s_tab, *s_sctab;
    load_tables(smem, s_tab, s_sctab);
    __syncthreads();
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < (1u << 24); k += gridDim.x * blockDim.x)
    {
        const float l = cl_logf_u(u32_to_randu(k << 8), s_tab);
        t[k] = l;
        t[GAUSS_OFF + k] = sqrtf(-2.0f * l);
    }
}

// Segment mode: decode tmin keys in place and sum npe per segment.
__global__ void finalize_segments(const uint32_t* maps, uint32_t* keys, int32_t* npe,
                                  int64_t n_seg, int32_t cells, const unsigned long long* steps,
                                  const unsigned int* err, unsigned long long* status)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t total = n_seg * cells;
    for (int64_t i = i0; i < total; i += stride) keys[i] = __float_as_uint(key_float(keys[i]));
    for (int64_t s = i0; s < n_seg; s += stride) {
        uint32_t acc = 0;
        const uint32_t* m = maps + s * cells;
        for (int c = 0; c < cells; ++c) acc += m[c];
        npe[s] = (int32_t)acc;
    }
    if (i0 == 0 && status) { status[0] = *steps; status[1] = *err; }
}

__global__ void decode_keys_kernel(uint32_t* keys, int64_t n)
{
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) keys[i] = __float_as_uint(key_float(keys[i]));
}

// ---- diagnostics ----
__global__ void debug_math_kernel(int fn, const float* in, float* out, int64_t n)
{
    __shared__ __align__(16) unsigned char tabs[LOGTAB_BYTES];
    double2 *s_tab, *s_sctab;
    load_tables(tabs, s_tab, s_sctab);
    __syncthreads();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const float x = in[i];
        float r;
        if (fn == 0) {
            r = cl_logf(x, s_tab);
        } else {
            float sv, cv;
            cl_sincosf(x, smem_addr(s_sctab), &sv, &cv);
            r = fn == 1 ? sv : cv;
        }
        out[i] = r;
    }
}

// The loop's quick decisions beside the exact expressions (items of `ni` input
// and `no` output floats):
//   7  x -> sqrt_mid(x)                       8  x -> rcp_mid(x)
//   9  (x, y, z, ux, uy, uz, Lx, Ly, Lz) -> quick distance and face (0: undecided), exact distance and face
//  10  (n1, n2, cosi, u) -> quick and exact "reflects" (total reflection included)
//  11  (u, d, length) -> 1 if the quick test rules a bulk event out, exact -length log u
//  12  as 9 -> quick face (0: undecided) and incidence cosine, the exact face's |direction|
__global__ void debug_step_kernel(int fn, const float* in, float* out, int64_t n)
{
    __shared__ __align__(16) unsigned char tabs[LOGTAB_BYTES];
    double2 *s_tab, *s_sctab;
    load_tables(tabs, s_tab, s_sctab);
    __syncthreads();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        if (fn == 7) out[i] = sqrt_mid(in[i]);
        if (fn == 8) out[i] = rcp_mid(in[i]);
        if (fn == 9) {
            const float* q = in + 9 * i;
            Physics P;
            P.L0 = q[6]; P.L1 = q[7]; P.L2 = q[8];
            float d, cosw;
            int32_t f;
            const bool ok = wall_hit_fast(P, q[0], q[1], q[2], q[3], q[4], q[5], d, f, cosw);
            out[4 * i] = d;
            out[4 * i + 1] = ok ? (float)f : 0.0f;
            out[4 * i + 3] = (float)wall_hit(P, q[0], q[1], q[2], q[3], q[4], q[5], d);
            out[4 * i + 2] = d;
        }
        if (fn == 12) {
            const float* q = in + 9 * i;
            Physics P;
            P.L0 = q[6]; P.L1 = q[7]; P.L2 = q[8];
            float d, cosw;
            int32_t f;
            const bool ok = wall_hit_fast(P, q[0], q[1], q[2], q[3], q[4], q[5], d, f, cosw);
            const int32_t g = wall_hit(P, q[0], q[1], q[2], q[3], q[4], q[5], d);
            out[3 * i] = ok ? (float)f : 0.0f;
            out[3 * i + 1] = cosw;
            out[3 * i + 2] = fabsf(g <= 2 ? q[3] : (g <= 4 ? q[4] : q[5]));
        }
        if (fn == 10) {
            const float* q = in + 4 * i;
            Physics P;
            P.n_crystal = q[0];
            P.fresnel_margin = fresnel_margin(q[0], q[1]);
            const float r = q[0] / q[1], sin2t = (r * r) * (1.0f - q[2] * q[2]);
            out[2 * i] = fresnel_reflects(P, q[1], sin2t, q[2], q[3]) ? 1.0f : 0.0f;
            out[2 * i + 1] = sin2t >= 1.0f || q[3] < fresnel_R(q[0], q[1], sin2t, q[2]) ? 1.0f : 0.0f;
        }
        if (fn == 11) {
            const float* q = in + 3 * i;
            out[2 * i] = q[0] < survive_below(q[1], survive_rate(q[2])) ? 1.0f : 0.0f;
            out[2 * i + 1] = (-q[2]) * cl_logf_u(q[0], s_tab);
        }
    }
}

__global__ void debug_philox_kernel(int use_curand, const uint32_t* ctr, uint32_t* out, int64_t n,
                                    uint32_t k0, uint32_t k1)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const uint4 c = make_uint4(ctr[4 * i], ctr[4 * i + 1], ctr[4 * i + 2], ctr[4 * i + 3]);
        uint4 o;
        if (use_curand) o = curand_Philox4x32_10(c, make_uint2(k0, k1));
        else o = philox4x32_10(c, k0, k1);
        out[4 * i] = o.x; out[4 * i + 1] = o.y; out[4 * i + 2] = o.z; out[4 * i + 3] = o.w;
    }
}

__global__ void debug_randu_kernel(float* out, int64_t n, int32_t n_per, uint32_t k0, uint32_t k1)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        SimpleStream s;
        const uint64_t pid = (uint64_t)i + 1ull;
        s.pid_lo = (uint32_t)pid; s.pid_hi = (uint32_t)(pid >> 32); s.block = 0; s.n = 0;
        s.b0 = s.b1 = s.b2 = s.b3 = 0;
        for (int32_t j = 0; j < n_per; ++j) out[i * n_per + j] = simple_randu(s, k0, k1);
    }
}

}  // namespace cl

// ===========================================================================
// Host side
// ===========================================================================
using namespace cl;

struct DevBuf {
    void* p = nullptr;
    size_t cap = 0;
};

// Calls on host arrays gather small ones in the handle's host buffer: one copy in
// and one out, with the steps and the error word, which the kernels leave behind
// the counters.  A copy to pageable memory waits for the stream by itself, and a
// point source's call ended in five of them.  2,000 CsI(Tl) photons from one point
// 237 -> 191 us a call, 10^6 784 -> 739 us (page-locked memory would save another
// 10 us and costs 400 us per handle).  Arrays beyond the limits (4,096 positions,
// 1,022 time bins, 507 segments), which belong to transports of milliseconds, are
// copied one by one, straight to the caller's memory.
constexpr size_t N_STATUS = sizeof(cl_counters) / 8, STATUS_BYTES = sizeof(cl_counters) + 16;
constexpr size_t STAGE_IN = 64 << 10, STAGE_OUT = 256 << 10;

struct cl_handle {
    int device = 0;
    int num_sms = 0;
    cudaStream_t stream = nullptr;
    DevBuf logtab;                 // the tables of the uniforms, or empty: the kernels compute them
    char err[512] = {0};
    DevBuf src, out, rec, scratch, dbg;
    char* stage = nullptr;         // STAGE_IN + STAGE_OUT bytes, or null: host arrays are copied one by one
    LaunchSetting launch;          // cl_set_launch
    int64_t last_steps = 0;
    int max_smem_optin = 0;
    int max_smem_per_sm = 0;
    unsigned long long budget_ns = (unsigned long long)(CL_DEFAULT_TIME_BUDGET_S * 1e9);
};

static thread_local char g_create_err[512];

__attribute__((format(printf, 3, 4)))
static int set_err(cl_handle* h, int code, const char* fmt, ...)
{
    if (h) {
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(h->err, sizeof h->err, fmt, ap);
        va_end(ap);
    }
    return code;
}

static int cuda_fail(cl_handle* h, cudaError_t e, const char* what)
{
    cudaGetLastError();  // clear sticky non-fatal error
    return set_err(h, e == cudaErrorMemoryAllocation ? CL_ERR_OOM : CL_ERR_CUDA,
                   "%s: %s", what, cudaGetErrorString(e));
}

#define CK(h, call, what)                                   \
    do {                                                    \
        cudaError_t e_ = (call);                            \
        if (e_ != cudaSuccess) return cuda_fail((h), e_, (what)); \
    } while (0)

static int ensure(cl_handle* h, DevBuf& b, size_t bytes)
{
    if (bytes <= b.cap) return CL_OK;
    if (b.p) { cudaFree(b.p); b.p = nullptr; b.cap = 0; }
    size_t want = bytes + bytes / 4 + 256;
    cudaError_t e = cudaMalloc(&b.p, want);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return set_err(h, CL_ERR_OOM, "device allocation of %zu bytes failed", want);
    }
    b.cap = want;
    return CL_OK;
}

static inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// Allow dynamic shared memory up to the opt-in limit minus the kernel's
// static shared memory (their sum may not exceed the limit).
template <int MODE, bool REC, bool TILE, int SPEC, bool TAB>
static void set_kernel_attrs_spec(int smem_optin)
{
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, transport_kernel<MODE, REC, TILE, SPEC, TAB>) != cudaSuccess) return;
    cudaFuncSetAttribute(transport_kernel<MODE, REC, TILE, SPEC, TAB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         smem_optin - (int)fa.sharedSizeBytes);
}

// Kernels that evaluate the logs in place serve the allocation-free entry point
// (point mode without records) in every configuration, and a handle whose
// tables could not be allocated in the general one.  One kernel for both carried
// the evaluation in the loop: scan 100.4 -> 98.0 ms, 3,001 events 20.6 -> 20.2 ms
// without it.
template <int MODE, bool REC>
constexpr bool spec_without_tables = MODE == POINT && !REC;
template <int MODE>
constexpr bool needs_tables = MODE >= SEGMENTS_CROWDED;

// Of the instances that a handle with (or without) the tables launches: the
// first call for an instance loads it.
template <int MODE, bool REC, bool TILE>
static void set_kernel_attrs(int smem_optin, bool tables)
{
    if (tables) {
        set_kernel_attrs_spec<MODE, REC, TILE, SPEC_ANY, true>(smem_optin);
        set_kernel_attrs_spec<MODE, REC, TILE, SPEC_ESR, true>(smem_optin);
        set_kernel_attrs_spec<MODE, REC, TILE, SPEC_TEFLON, true>(smem_optin);
        return;
    }
    if constexpr (!needs_tables<MODE>) set_kernel_attrs_spec<MODE, REC, TILE, SPEC_ANY, false>(smem_optin);
    if constexpr (spec_without_tables<MODE, REC>) {
        set_kernel_attrs_spec<MODE, REC, TILE, SPEC_ESR, false>(smem_optin);
        set_kernel_attrs_spec<MODE, REC, TILE, SPEC_TEFLON, false>(smem_optin);
    }
}

extern "C" {

const char* cl_version(void) { return CL_VERSION_STRING; }
int cl_abi_version(void) { return CL_ABI_VERSION; }

int cl_create(cl_handle** out, int device)
{
    g_create_err[0] = 0;
    if (!out) {
        snprintf(g_create_err, sizeof g_create_err, "cl_create: null output pointer");
        return CL_ERR_ARG;
    }
    *out = nullptr;
    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess || device < 0 || device >= ndev) {
        cudaGetLastError();
        snprintf(g_create_err, sizeof g_create_err, "cl_create: CUDA device %d unavailable (%s)",
                 device, e != cudaSuccess ? cudaGetErrorString(e) : "no such device");
        return e != cudaSuccess ? CL_ERR_CUDA : CL_ERR_ARG;
    }
    cl_handle* h = new (std::nothrow) cl_handle();
    if (!h) {
        snprintf(g_create_err, sizeof g_create_err, "cl_create: out of host memory");
        return CL_ERR_OOM;
    }
    h->device = device;
    e = cudaSetDevice(device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&h->num_sms, cudaDevAttrMultiProcessorCount, device);
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&h->max_smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&h->max_smem_per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
        cudaGetLastError();
        snprintf(g_create_err, sizeof g_create_err, "cl_create: %s", cudaGetErrorString(e));
        delete h;
        return CL_ERR_CUDA;
    }
    if (ensure(h, h->scratch, 64) != CL_OK) {
        snprintf(g_create_err, sizeof g_create_err, "cl_create: %s", h->err);
        cudaStreamDestroy(h->stream);
        delete h;
        return CL_ERR_OOM;
    }
    h->stage = (char*)malloc(STAGE_IN + STAGE_OUT);
    // 128 MB: the logs of all 2^24 uniforms and their sqrt(-2 log u); without
    // them (allocation failure) the kernels evaluate the same functions in place.
    // The logs alone, and the root in the loop (sqrt_mid, the same bits), would fit
    // L2 beside everything else, and cost more: scan 92.6 -> 93.9 ms, 2,000 photons
    // 208 -> 223 us, 3,001 events 18.83 -> 18.87 ms.  A handle takes 0.8 ms to make
    // with either.
    if (cudaMalloc(&h->logtab.p, sizeof(float) << 25) == cudaSuccess) {
        h->logtab.cap = sizeof(float) << 25;
        logtab_fill<<<h->num_sms * 4, 256, LOGTAB_BYTES, h->stream>>>((float*)h->logtab.p);
        if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(h->stream) != cudaSuccess) {
            cudaGetLastError();
            cudaFree(h->logtab.p);
            h->logtab = DevBuf();
        }
    } else {
        cudaGetLastError();
        h->logtab = DevBuf();
    }
    const bool tables = h->logtab.p != nullptr;
    set_kernel_attrs<POINT, false, true>(h->max_smem_optin, tables);
    set_kernel_attrs<POINT, true, true>(h->max_smem_optin, tables);
    set_kernel_attrs<POINT, false, false>(h->max_smem_optin, tables);
    set_kernel_attrs<POINT, true, false>(h->max_smem_optin, tables);
    set_kernel_attrs<SEGMENTS, false, false>(h->max_smem_optin, tables);
    set_kernel_attrs<SEGMENTS, true, false>(h->max_smem_optin, tables);
    set_kernel_attrs<MOMENTS, false, false>(h->max_smem_optin, tables);
    set_kernel_attrs<SEGMENTS_CROWDED, false, false>(h->max_smem_optin, tables);
    set_kernel_attrs<SEGMENTS_CROWDED, true, false>(h->max_smem_optin, tables);
    set_kernel_attrs<MOMENTS_CROWDED, false, false>(h->max_smem_optin, tables);
    cudaGetLastError();
    *out = h;
    return CL_OK;
}

void cl_destroy(cl_handle* h)
{
    if (!h) return;
    cudaSetDevice(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    DevBuf* bufs[] = {&h->src, &h->out, &h->rec, &h->scratch, &h->dbg, &h->logtab};
    for (DevBuf* b : bufs) if (b->p) cudaFree(b->p);
    free(h->stage);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
}

const char* cl_last_error(const cl_handle* h) { return h ? h->err : g_create_err; }

int64_t cl_last_steps(const cl_handle* h) { return h ? h->last_steps : 0; }

int cl_set_launch(cl_handle* h, int ctas_per_sm, int threads_per_cta, int warp_chunk)
{
    if (!h) return CL_ERR_STATE;
    if (ctas_per_sm < 0 || ctas_per_sm > 32) return set_err(h, CL_ERR_ARG, "ctas_per_sm out of range");
    if (threads_per_cta != 0 && (threads_per_cta < 32 || threads_per_cta > 256 || threads_per_cta % 32))
        return set_err(h, CL_ERR_ARG, "threads_per_cta must be a multiple of 32 in [32, 256]");
    if (warp_chunk != 0 && (warp_chunk < 32 || warp_chunk > (1 << 20)))
        return set_err(h, CL_ERR_ARG, "warp_chunk must be in [32, 2^20]");
    h->launch.ctas_per_sm = ctas_per_sm;
    h->launch.threads = threads_per_cta;
    h->launch.warp_chunk = warp_chunk;
    return CL_OK;
}

int cl_set_time_budget(cl_handle* h, double seconds)
{
    if (!h) return CL_ERR_STATE;
    if (!(seconds >= 0.0) || !std::isfinite(seconds) || seconds > 1.0e9)
        return set_err(h, CL_ERR_ARG, "time budget must be finite, >= 0 and <= 1e9 s");
    h->budget_ns = (unsigned long long)(seconds * 1e9);
    return CL_OK;
}

}  // extern "C"

// ---- argument validation shared by the entry points ----
static int check_params(cl_handle* h, const cl_box* box, const cl_optical_params* op,
                        const cl_readout* ro, const cl_time_binning* tb, float tau_ns,
                        int32_t max_bounces)
{
    if (!box || !op || !ro || !tb) return set_err(h, CL_ERR_ARG, "null parameter struct");
    if (max_bounces > CL_MAX_BOUNCES_LIMIT)
        return set_err(h, CL_ERR_ARG, "max_bounces %d above the limit %d", (int)max_bounces,
                       (int)CL_MAX_BOUNCES_LIMIT);
    for (int i = 0; i < 3; ++i)
        if (!(box->L[i] > 0.0f) || !std::isfinite(box->L[i]))
            return set_err(h, CL_ERR_ARG, "box sizes must be finite and positive");
    if (ro->grid.nx < 1 || ro->grid.ny < 1 || (int64_t)ro->grid.nx * ro->grid.ny > 32767)
        return set_err(h, CL_ERR_ARG, "SiPM grid must have 1 <= nx*ny <= 32767");
    if (!(ro->grid.pitch_mm > 0.0f)) return set_err(h, CL_ERR_ARG, "pitch_mm must be positive");
    if (tb->nbins < 0 || tb->nbins > (1 << 24) || !(tb->bin_ns > 0.0f))
        return set_err(h, CL_ERR_ARG, "time binning needs bin_ns > 0 and 0 <= nbins <= 2^24");
    if (!(op->n_crystal > 0.0f) || !(op->n_coupling > 0.0f))
        return set_err(h, CL_ERR_ARG, "refractive indices must be positive");
    if (std::isnan(op->abs_len_mm) || std::isnan(op->rayleigh_mm) || std::isnan(op->wrap_R) ||
        std::isnan(op->sigma_alpha) || std::isnan(op->pde) || std::isnan(tau_ns) || std::isinf(tau_ns))
        return set_err(h, CL_ERR_ARG, "NaN/Inf in optical parameters or tau_ns");
    return CL_OK;
}

static Physics make_physics(const cl_box* box, const cl_optical_params* op, const cl_readout* ro,
                            const cl_time_binning* tb, float tau_ns, int32_t max_bounces, uint64_t seed)
{
    Physics P;
    memset(&P, 0, sizeof P);
    P.L0 = box->L[0]; P.L1 = box->L[1]; P.L2 = box->L[2];
    P.n_crystal = op->n_crystal; P.n_coupling = op->n_coupling;
    P.abs_len = op->abs_len_mm; P.ray_len = op->rayleigh_mm;
    P.wrap_R = op->wrap_R; P.sigma_alpha = op->sigma_alpha; P.pde = op->pde;
    P.inv_v = op->n_crystal / 299.792458f;
    P.cx = ro->cx; P.cy = ro->cy; P.r2 = ro->r2; P.sur_R = ro->sur_R;
    P.pitch = ro->grid.pitch_mm; P.bin_ns = tb->bin_ns; P.tau = tau_ns;
    P.nx = ro->grid.nx; P.ny = ro->grid.ny; P.nbins = tb->nbins; P.max_bounces = max_bounces;
    P.key0 = (uint32_t)seed; P.key1 = (uint32_t)(seed >> 32);
    {
        uint32_t k0 = P.key0, k1 = P.key1;
        for (int r = 0; r < 10; ++r) {
            P.rk[2 * r] = k0; P.rk[2 * r + 1] = k1;
            k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
        }
        const float qc = op->n_crystal / op->n_coupling;   // IEEE division on the host, as on the device
        const float qa = op->n_crystal / 1.0f;
        P.qc2 = qc * qc;
        P.qa2 = qa * qa;
    }
    P.abs_rate = survive_rate(op->abs_len_mm);
    P.ray_rate = survive_rate(op->rayleigh_mm);
    P.fresnel_margin = fresnel_margin(op->n_crystal, op->n_coupling);
    P.abs_finite = std::isfinite(op->abs_len_mm) ? 1 : 0;
    P.ray_finite = std::isfinite(op->rayleigh_mm) ? 1 : 0;
    P.wrap_specular = op->wrap_specular ? 1 : 0;
    P.air_gap = op->air_gap ? 1 : 0;
    P.disc = ro->disc ? 1 : 0;
    P.sur_specular = ro->sur_specular ? 1 : 0;
    P.two_sided = ro->two_sided ? 1 : 0;
    return P;
}

// Scratch words: [0] queue u64, [1] steps u64, [2] done u32 | err u32
struct Scratch {
    unsigned long long* queue;
    unsigned long long* steps;
    unsigned int* done;
    unsigned int* err;
};

static Scratch scratch_of(cl_handle* h)
{
    unsigned long long* base = (unsigned long long*)h->scratch.p;
    Scratch s;
    s.queue = base;
    s.steps = base + 1;
    s.done = (unsigned int*)(base + 2);
    s.err = s.done + 1;
    return s;
}

// The compiled configuration a launch can use (SPEC_ANY where none matches).
static int spec_of(const Physics& P)
{
    if (!P.air_gap || !(P.sigma_alpha > 0.0f) || P.disc || P.two_sided || !P.abs_finite || !P.ray_finite ||
        P.abs_len < 0.0f || P.ray_len < 0.0f)
        return SPEC_ANY;
    return P.wrap_specular ? SPEC_ESR : SPEC_TEFLON;
}

template <int MODE, bool REC, bool TILE, int SPEC, bool TAB>
static int launch_transport_spec(cl_handle* h, const KArgs& a, size_t smem, cudaStream_t st)
{
    auto kern = transport_kernel<MODE, REC, TILE, SPEC, TAB>;
    int per_sm = 0;
    CK(h, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, h->launch.threads ? h->launch.threads : AUTO_THREADS,
                                                        smem), "occupancy");
    if (per_sm < 1) return set_err(h, CL_ERR_ARG, "transport kernel does not fit on an SM (shared tile too large)");
    const LaunchShape shape = launch_shape(a.n, h->num_sms, per_sm, h->launch);
    KArgs b = a;
    b.warp_chunk = shape.warp_chunk;
    kern<<<(unsigned)shape.grid, shape.threads, smem, st>>>(b);
    CK(h, cudaGetLastError(), "transport kernel launch");
    return CL_OK;
}

template <int MODE, bool REC, bool TILE>
static int launch_transport(cl_handle* h, const KArgs& a, size_t smem, cudaStream_t st)
{
    const int spec = spec_of(a.P);
    if constexpr (!needs_tables<MODE>) {
        if (!a.logtab) {
            if constexpr (spec_without_tables<MODE, REC>) {
                if (spec == SPEC_ESR) return launch_transport_spec<MODE, REC, TILE, SPEC_ESR, false>(h, a, smem, st);
                if (spec == SPEC_TEFLON) return launch_transport_spec<MODE, REC, TILE, SPEC_TEFLON, false>(h, a, smem, st);
            }
            return launch_transport_spec<MODE, REC, TILE, SPEC_ANY, false>(h, a, smem, st);
        }
    }
    switch (spec) {
    case SPEC_ESR: return launch_transport_spec<MODE, REC, TILE, SPEC_ESR, true>(h, a, smem, st);
    case SPEC_TEFLON: return launch_transport_spec<MODE, REC, TILE, SPEC_TEFLON, true>(h, a, smem, st);
    default: return launch_transport_spec<MODE, REC, TILE, SPEC_ANY, true>(h, a, smem, st);
    }
}

static int enqueue_point(cl_handle* h, const Physics& P, const float* px, const float* py,
                         const float* pz, const float* pt, int32_t npos, int64_t n, uint64_t pid0,
                         uint32_t* counts, uint32_t* keys, unsigned long long* counters,
                         const cl_records* rec, cudaStream_t st, unsigned long long* status = nullptr)
{
    const int cells = P.nx * P.ny;
    const int bins_total = P.nbins + 1;
    const int64_t n_counts = (int64_t)cells * bins_total;
    Scratch s = scratch_of(h);
    init_kernel<<<(unsigned)std::min<int64_t>((n_counts + 255) / 256 + 1, 4096), 256, 0, st>>>(
        counts, n_counts, keys, cells, counters, s.queue, s.steps, s.done, s.err);
    CK(h, cudaGetLastError(), "init kernel launch");
    if (n == 0) {
        // no photons: decode the +Inf keys into Float32 +Inf
        if (status) CK(h, cudaMemsetAsync(status, 0, 2 * sizeof *status, st), "zero status");
        decode_keys_kernel<<<1, 256, 0, st>>>(keys, cells);
        CK(h, cudaGetLastError(), "decode launch");
        return CL_OK;
    }
    KArgs a;
    memset(&a, 0, sizeof a);
    a.P = P; a.pid0 = pid0; a.n = n; a.npos = npos;
    a.cells = cells; a.bins_total = bins_total;
    a.px = px; a.py = py; a.pz = pz; a.pt = pt;
    a.counts = counts; a.keys = keys; a.counters = counters;
    const bool want_rec = rec && (rec->status || rec->idx || rec->t || rec->bounces);
    if (want_rec) { a.r_status = rec->status; a.r_idx = rec->idx; a.r_t = rec->t; a.r_bounces = rec->bounces; }
    a.queue = s.queue; a.steps = s.steps; a.done = s.done; a.err = s.err; a.status = status;
    a.logtab = (const float*)h->logtab.p;
    a.budget_ns = h->budget_ns;
    const size_t tile_bytes = ((size_t)n_counts + cells) * sizeof(uint32_t);
    const size_t base_bytes = LOGTAB_BYTES + RING_BYTES;
    // the shared-memory histogram tile only where it still leaves room for 4
    // CTAs per SM: with fewer resident warps the loop issues less often, which
    // costs more than the tile saves in global atomics (CsI(Tl), 4M photons, 8x8x81
    // bins: 1,867 us on global atomics at 4 CTAs/SM, 2,038 with the tile at 3; 10^6
    // photons 728 and 751).  Room for 3 where the photons in flight (more than
    // 2^17) share few slots, because the bins that the decay time reaches are few:
    // there the reductions on one address are the bound (the same with no decay
    // time: 2,040 and 1,950; a clear crystal, 41 to 81 bins: 1,865 and 860 to 910;
    // 75 to 108 slots, most photons gone after a step: 590 and 340, after twelve:
    // 1,860 and 1,930).
    const double slots = (double)cells * (1.0 + (P.tau > 0.0f ? std::floor((double)P.tau / (double)P.bin_ns) : 0.0));
    const int ctas = slots <= 128.0 && n >= (1 << 17) ? 3 : 4;
    const size_t per_cta = base_bytes + tile_bytes + CTA_EXTRA_SMEM;
    const bool tile = base_bytes + tile_bytes <= (size_t)std::min(h->max_smem_optin, 160 * 1024) &&
                      ctas * per_cta <= (size_t)h->max_smem_per_sm;
    const size_t smem = base_bytes + (tile ? tile_bytes : 0);
    if (tile) return want_rec ? launch_transport<POINT, true, true>(h, a, smem, st)
                              : launch_transport<POINT, false, true>(h, a, smem, st);
    return want_rec ? launch_transport<POINT, true, false>(h, a, smem, st)
                    : launch_transport<POINT, false, false>(h, a, smem, st);
}

static int enqueue_segments(cl_handle* h, const Physics& P, const float* sx, const float* sy,
                            const float* sz, const float* sT, const int64_t* off, const int32_t* segid,
                            int64_t n_src, int64_t n_seg, int64_t n, uint64_t pid0,
                            uint32_t* maps, uint32_t* keys, int32_t* npe,
                            unsigned long long* counters, const cl_records* rec, cudaStream_t st,
                            unsigned long long* tsum = nullptr, unsigned long long* tsum2 = nullptr,
                            const SurSampleArgs* sample = nullptr, unsigned long long* status = nullptr)
{
    const int cells = P.nx * P.ny;
    const int64_t total = (int64_t)cells * n_seg;
    Scratch s = scratch_of(h);
    init_kernel<<<(unsigned)std::min<int64_t>((total + 255) / 256 + 1, 8192), 256, 0, st>>>(
        maps, total, keys, total, counters, s.queue, s.steps, s.done, s.err);
    CK(h, cudaGetLastError(), "init kernel launch");
    const bool moments = tsum && tsum2;
    if (moments) {
        CK(h, cudaMemsetAsync(tsum, 0, (size_t)total * sizeof(unsigned long long), st), "zero moments");
        CK(h, cudaMemsetAsync(tsum2, 0, (size_t)total * sizeof(unsigned long long), st), "zero moments");
    }
    if (n > 0) {
        KArgs a;
        memset(&a, 0, sizeof a);
        a.P = P; a.pid0 = pid0; a.n = n; a.npos = 1;
        a.cells = cells; a.bins_total = P.nbins + 1;
        a.px = sx; a.py = sy; a.pz = sz; a.pt = sT;
        a.src_off = off; a.src_seg = segid; a.n_src = n_src; a.n_seg = n_seg;
        a.keys = keys; a.maps = maps; a.counters = counters;
        const bool want_rec = rec && (rec->status || rec->idx || rec->t || rec->bounces);
        if (want_rec) { a.r_status = rec->status; a.r_idx = rec->idx; a.r_t = rec->t; a.r_bounces = rec->bounces; }
        a.queue = s.queue; a.steps = s.steps; a.done = s.done; a.err = s.err;
        a.logtab = (const float*)h->logtab.p;
        a.budget_ns = h->budget_ns;
        const size_t smem = LOGTAB_BYTES + RING_BYTES;
        a.tsum = tsum; a.tsum2 = tsum2;
        const bool crowded = n / total >= (cells < 64 ? CROWDED_FEW : CROWDED) && total <= (int64_t)UINT32_MAX && a.logtab;
        const int rc = crowded ? (moments ? launch_transport<MOMENTS_CROWDED, false, false>(h, a, smem, st)
                                  : want_rec ? launch_transport<SEGMENTS_CROWDED, true, false>(h, a, smem, st)
                                             : launch_transport<SEGMENTS_CROWDED, false, false>(h, a, smem, st))
                     : moments ? launch_transport<MOMENTS, false, false>(h, a, smem, st)
                     : want_rec ? launch_transport<SEGMENTS, true, false>(h, a, smem, st)
                                : launch_transport<SEGMENTS, false, false>(h, a, smem, st);
        if (rc != CL_OK) return rc;
    }
    if (sample) {
        SurSampleArgs sa = *sample;
        sa.maps = maps; sa.keys = keys; sa.err = s.err;
        CK(h, launch_surrogate_sample(sa, h->num_sms, st), "surrogate sampler launch");
    }
    finalize_segments<<<(unsigned)std::min<int64_t>((total + 255) / 256 + 1, 8192), 256, 0, st>>>(
        maps, keys, npe, n_seg, cells, s.steps, s.err, status);
    CK(h, cudaGetLastError(), "finalize launch");
    return CL_OK;
}

static int report(cl_handle* h, unsigned long long steps, unsigned int err)
{
    h->last_steps = (int64_t)steps;
    if (err & 32u)
        return set_err(h, CL_ERR_TIMEOUT, "the transport ran past the handle's time budget (%.3g s); "
                       "its outputs are incomplete", (double)h->budget_ns * 1e-9);
    if (err & 2u) return set_err(h, CL_ERR_CUDA, "internal error: uniform ring underflow in the transport kernel");
    if (err & 16u) return set_err(h, CL_ERR_ARG, "a source's segment id is out of range (its detections were dropped)");
    if (err & 8u) return set_err(h, CL_ERR_ARG, "a surrogate site's segment id is out of range (site skipped)");
    if (err & 4u) return set_err(h, CL_ERR_TIMEOUT, "a loop budget of the surrogate sampler ran out");
    if (err) return set_err(h, CL_ERR_TIMEOUT, "a device-side loop budget ran out (Rayleigh rejection sampler)");
    return CL_OK;
}

static int collect(cl_handle* h, cudaStream_t st)
{
    unsigned long long words[3];     // the scratch words
    CK(h, cudaMemcpyAsync(words, h->scratch.p, sizeof words, cudaMemcpyDeviceToHost, st), "copy status");
    CK(h, cudaStreamSynchronize(st), "stream synchronize");
    return report(h, words[1], (unsigned int)(words[2] >> 32));
}

extern "C" {

int cl_run_photons(cl_handle* h, const cl_box* box, const cl_optical_params* op,
                   const cl_readout* ro, const cl_time_binning* tb,
                   const float* px, const float* py, const float* pz,
                   const float* pt, int32_t npos,
                   int64_t n_photons, uint64_t seed, uint64_t pid_offset,
                   float tau_ns, int32_t max_bounces,
                   uint32_t* counts, float* first_ns, cl_counters* counters,
                   const cl_records* records)
{
    if (!h) return CL_ERR_STATE;
    h->err[0] = 0;
    int rc = check_params(h, box, op, ro, tb, tau_ns, max_bounces);
    if (rc != CL_OK) return rc;
    if (npos < 1 || !px || !py || !pz) return set_err(h, CL_ERR_ARG, "need npos >= 1 source positions");
    if (n_photons < 0) return set_err(h, CL_ERR_ARG, "n_photons must be >= 0");
    if (!counts || !first_ns || !counters) return set_err(h, CL_ERR_ARG, "null output buffer");
    CK(h, cudaSetDevice(h->device), "cudaSetDevice");
    cudaStream_t st = h->stream;

    const int cells = ro->grid.nx * ro->grid.ny;
    const size_t n_counts = (size_t)cells * (size_t)(tb->nbins + 1);
    // device layout: sources | counts | keys | counters ; records separately
    const size_t b_src = align256(4 * (size_t)npos * sizeof(float));
    const size_t b_counts = align256(n_counts * sizeof(uint32_t));
    const size_t b_keys = align256((size_t)cells * sizeof(uint32_t));
    const size_t b_ctr = align256(STATUS_BYTES);
    if ((rc = ensure(h, h->src, b_src)) != CL_OK) return rc;
    if ((rc = ensure(h, h->out, b_counts + b_keys + b_ctr)) != CL_OK) return rc;
    float* d_px = (float*)h->src.p;
    float* d_py = d_px + npos;
    float* d_pz = d_py + npos;
    float* d_pt = d_pz + npos;
    uint32_t* d_counts = (uint32_t*)h->out.p;
    uint32_t* d_keys = (uint32_t*)((char*)h->out.p + b_counts);
    unsigned long long* d_ctr = (unsigned long long*)((char*)h->out.p + b_counts + b_keys);

    cl_records drec;
    memset(&drec, 0, sizeof drec);
    const bool want_rec = records && (records->status || records->idx || records->t || records->bounces);
    if (want_rec && n_photons > 0) {
        const size_t n = (size_t)n_photons;
        const size_t b1 = align256(n), b2 = align256(2 * n), b4 = align256(4 * n);
        if ((rc = ensure(h, h->rec, b1 + b2 + 2 * b4)) != CL_OK) return rc;
        char* base = (char*)h->rec.p;
        if (records->status) drec.status = (uint8_t*)base;
        if (records->idx) drec.idx = (int16_t*)(base + b1);
        if (records->t) drec.t = (float*)(base + b1 + b2);
        if (records->bounces) drec.bounces = (int32_t*)(base + b1 + b2 + b4);
    }

    const size_t fs = (size_t)npos * sizeof(float);
    if (h->stage && 4 * fs <= STAGE_IN) {
        char* in = h->stage;
        memcpy(in, px, fs);
        memcpy(in + fs, py, fs);
        memcpy(in + 2 * fs, pz, fs);
        if (pt) memcpy(in + 3 * fs, pt, fs);
        CK(h, cudaMemcpyAsync(d_px, in, (pt ? 4 : 3) * fs, cudaMemcpyHostToDevice, st), "copy positions");
    } else {
        CK(h, cudaMemcpyAsync(d_px, px, fs, cudaMemcpyHostToDevice, st), "copy px");
        CK(h, cudaMemcpyAsync(d_py, py, fs, cudaMemcpyHostToDevice, st), "copy py");
        CK(h, cudaMemcpyAsync(d_pz, pz, fs, cudaMemcpyHostToDevice, st), "copy pz");
        if (pt) CK(h, cudaMemcpyAsync(d_pt, pt, fs, cudaMemcpyHostToDevice, st), "copy pt");
    }

    const Physics P = make_physics(box, op, ro, tb, tau_ns, max_bounces, seed);
    rc = enqueue_point(h, P, d_px, d_py, d_pz, pt ? d_pt : nullptr, npos, n_photons, pid_offset,
                       d_counts, d_keys, d_ctr, want_rec ? &drec : nullptr, st, d_ctr + N_STATUS);
    if (rc != CL_OK) return rc;

    char* const back = h->stage ? h->stage + STAGE_IN : nullptr;
    const bool gathered = h->stage && b_counts + b_keys + b_ctr <= STAGE_OUT;
    if (gathered) {
        CK(h, cudaMemcpyAsync(back, h->out.p, b_counts + b_keys + STATUS_BYTES, cudaMemcpyDeviceToHost, st),
           "copy outputs");
    } else {
        CK(h, cudaMemcpyAsync(counts, d_counts, n_counts * sizeof(uint32_t), cudaMemcpyDeviceToHost, st), "copy counts");
        CK(h, cudaMemcpyAsync(first_ns, d_keys, (size_t)cells * sizeof(float), cudaMemcpyDeviceToHost, st), "copy first_ns");
        CK(h, cudaMemcpyAsync(counters, d_ctr, sizeof(cl_counters), cudaMemcpyDeviceToHost, st), "copy counters");
    }
    if (want_rec && n_photons > 0) {
        const size_t n = (size_t)n_photons;
        if (records->status) CK(h, cudaMemcpyAsync(records->status, drec.status, n, cudaMemcpyDeviceToHost, st), "copy status");
        if (records->idx) CK(h, cudaMemcpyAsync(records->idx, drec.idx, 2 * n, cudaMemcpyDeviceToHost, st), "copy idx");
        if (records->t) CK(h, cudaMemcpyAsync(records->t, drec.t, 4 * n, cudaMemcpyDeviceToHost, st), "copy t");
        if (records->bounces) CK(h, cudaMemcpyAsync(records->bounces, drec.bounces, 4 * n, cudaMemcpyDeviceToHost, st), "copy bounces");
    }
    if (!gathered) return collect(h, st);
    CK(h, cudaStreamSynchronize(st), "stream synchronize");
    unsigned long long status[2];
    memcpy(counts, back, n_counts * sizeof(uint32_t));
    memcpy(first_ns, back + b_counts, (size_t)cells * sizeof(float));
    memcpy(counters, back + b_counts + b_keys, sizeof(cl_counters));
    memcpy(status, back + b_counts + b_keys + 8 * N_STATUS, sizeof status);
    return report(h, status[0], (unsigned int)status[1]);
}

int cl_run_photons_device(cl_handle* h, const cl_box* box, const cl_optical_params* op,
                          const cl_readout* ro, const cl_time_binning* tb,
                          const float* d_px, const float* d_py, const float* d_pz,
                          const float* d_pt, int32_t npos,
                          int64_t n_photons, uint64_t seed, uint64_t pid_offset,
                          float tau_ns, int32_t max_bounces,
                          uint32_t* d_counts, float* d_first_ns,
                          cl_counters* d_counters, const cl_records* d_records, void* stream)
{
    if (!h) return CL_ERR_STATE;
    h->err[0] = 0;
    int rc = check_params(h, box, op, ro, tb, tau_ns, max_bounces);
    if (rc != CL_OK) return rc;
    if (npos < 1 || !d_px || !d_py || !d_pz) return set_err(h, CL_ERR_ARG, "need npos >= 1 source positions");
    if (n_photons < 0) return set_err(h, CL_ERR_ARG, "n_photons must be >= 0");
    if (!d_counts || !d_first_ns || !d_counters) return set_err(h, CL_ERR_ARG, "null output buffer");
    CK(h, cudaSetDevice(h->device), "cudaSetDevice");
    cudaStream_t st = stream ? (cudaStream_t)stream : h->stream;
    const Physics P = make_physics(box, op, ro, tb, tau_ns, max_bounces, seed);
    return enqueue_point(h, P, d_px, d_py, d_pz, d_pt, npos, n_photons, pid_offset, d_counts,
                         (uint32_t*)d_first_ns, (unsigned long long*)d_counters, d_records, st);
}

static int check_segments(cl_handle* h, const int64_t* off, const int32_t* seg, int64_t n_src,
                          int64_t n_seg, int64_t* total)
{
    if (n_src < 1 || n_seg < 1) return set_err(h, CL_ERR_ARG, "need n_src >= 1 and n_segments >= 1");
    if (!off || !seg) return set_err(h, CL_ERR_ARG, "null source offsets or segment ids");
    if (off[0] != 0) return set_err(h, CL_ERR_ARG, "src_offsets[0] must be 0");
    for (int64_t s = 0; s < n_src; ++s) {
        if (off[s + 1] < off[s]) return set_err(h, CL_ERR_ARG, "src_offsets must be non-decreasing");
        if (seg[s] < 0 || seg[s] >= n_seg) return set_err(h, CL_ERR_ARG, "segment id out of range");
        if (s > 0 && seg[s] < seg[s - 1]) return set_err(h, CL_ERR_ARG, "segment ids must be non-decreasing");
    }
    *total = off[n_src];
    return CL_OK;
}

int cl_run_segments(cl_handle* h, const cl_box* box, const cl_optical_params* op,
                    const cl_readout* ro, const cl_time_binning* tb,
                    const float* sx, const float* sy, const float* sz,
                    const float* st_, const int64_t* src_offsets,
                    const int32_t* src_segment, int64_t n_src, int64_t n_segments,
                    uint64_t seed, uint64_t pid_offset,
                    float tau_ns, int32_t max_bounces,
                    uint32_t* maps, float* tmin, int32_t* npe,
                    cl_counters* counters, const cl_records* records)
{
    if (!h) return CL_ERR_STATE;
    h->err[0] = 0;
    int rc = check_params(h, box, op, ro, tb, tau_ns, max_bounces);
    if (rc != CL_OK) return rc;
    int64_t n = 0;
    if ((rc = check_segments(h, src_offsets, src_segment, n_src, n_segments, &n)) != CL_OK) return rc;
    if (!sx || !sy || !sz) return set_err(h, CL_ERR_ARG, "null source positions");
    if (!maps || !tmin || !npe || !counters) return set_err(h, CL_ERR_ARG, "null output buffer");
    CK(h, cudaSetDevice(h->device), "cudaSetDevice");
    cudaStream_t st = h->stream;
    const int cells = ro->grid.nx * ro->grid.ny;
    const size_t total = (size_t)cells * (size_t)n_segments;
    const size_t b_f = align256((size_t)n_src * sizeof(float));
    const size_t b_off = align256((size_t)(n_src + 1) * sizeof(int64_t));
    const size_t b_seg = align256((size_t)n_src * sizeof(int32_t));
    const size_t b_maps = align256(total * sizeof(uint32_t));
    const size_t b_npe = align256((size_t)n_segments * sizeof(int32_t));
    const size_t b_ctr = align256(STATUS_BYTES);
    if ((rc = ensure(h, h->src, 4 * b_f + b_off + b_seg)) != CL_OK) return rc;
    if ((rc = ensure(h, h->out, 2 * b_maps + b_npe + b_ctr)) != CL_OK) return rc;
    char* sb = (char*)h->src.p;
    float* d_sx = (float*)sb;
    float* d_sy = (float*)(sb + b_f);
    float* d_sz = (float*)(sb + 2 * b_f);
    float* d_st = (float*)(sb + 3 * b_f);
    int64_t* d_off = (int64_t*)(sb + 4 * b_f);
    int32_t* d_seg = (int32_t*)(sb + 4 * b_f + b_off);
    char* ob = (char*)h->out.p;
    uint32_t* d_maps = (uint32_t*)ob;
    uint32_t* d_keys = (uint32_t*)(ob + b_maps);
    int32_t* d_npe = (int32_t*)(ob + 2 * b_maps);
    unsigned long long* d_ctr = (unsigned long long*)(ob + 2 * b_maps + b_npe);

    cl_records drec;
    memset(&drec, 0, sizeof drec);
    const bool want_rec = records && (records->status || records->idx || records->t || records->bounces);
    if (want_rec && n > 0) {
        const size_t m = (size_t)n;
        const size_t b1 = align256(m), b2 = align256(2 * m), b4 = align256(4 * m);
        if ((rc = ensure(h, h->rec, b1 + b2 + 2 * b4)) != CL_OK) return rc;
        char* base = (char*)h->rec.p;
        if (records->status) drec.status = (uint8_t*)base;
        if (records->idx) drec.idx = (int16_t*)(base + b1);
        if (records->t) drec.t = (float*)(base + b1 + b2);
        if (records->bounces) drec.bounces = (int32_t*)(base + b1 + b2 + b4);
    }
    const size_t fs = (size_t)n_src * sizeof(float), os = (size_t)(n_src + 1) * sizeof(int64_t);
    const size_t ss = (size_t)n_src * sizeof(int32_t);
    if (h->stage && 4 * b_f + b_off + b_seg <= STAGE_IN) {
        char* in = h->stage;              // laid out as on the device
        memcpy(in, sx, fs);
        memcpy(in + b_f, sy, fs);
        memcpy(in + 2 * b_f, sz, fs);
        if (st_) memcpy(in + 3 * b_f, st_, fs);
        memcpy(in + 4 * b_f, src_offsets, os);
        memcpy(in + 4 * b_f + b_off, src_segment, ss);
        CK(h, cudaMemcpyAsync(sb, in, 4 * b_f + b_off + ss, cudaMemcpyHostToDevice, st), "copy sources");
    } else {
        CK(h, cudaMemcpyAsync(d_sx, sx, fs, cudaMemcpyHostToDevice, st), "copy sx");
        CK(h, cudaMemcpyAsync(d_sy, sy, fs, cudaMemcpyHostToDevice, st), "copy sy");
        CK(h, cudaMemcpyAsync(d_sz, sz, fs, cudaMemcpyHostToDevice, st), "copy sz");
        if (st_) CK(h, cudaMemcpyAsync(d_st, st_, fs, cudaMemcpyHostToDevice, st), "copy st");
        CK(h, cudaMemcpyAsync(d_off, src_offsets, os, cudaMemcpyHostToDevice, st), "copy offsets");
        CK(h, cudaMemcpyAsync(d_seg, src_segment, ss, cudaMemcpyHostToDevice, st), "copy segments");
    }

    const Physics P = make_physics(box, op, ro, tb, tau_ns, max_bounces, seed);
    rc = enqueue_segments(h, P, d_sx, d_sy, d_sz, st_ ? d_st : nullptr, d_off, d_seg, n_src, n_segments,
                          n, pid_offset, d_maps, d_keys, d_npe, d_ctr, want_rec ? &drec : nullptr, st, nullptr, nullptr,
                          nullptr, d_ctr + N_STATUS);
    if (rc != CL_OK) return rc;
    char* const back = h->stage ? h->stage + STAGE_IN : nullptr;
    const bool gathered = h->stage && 2 * b_maps + b_npe + b_ctr <= STAGE_OUT;
    if (gathered) {
        CK(h, cudaMemcpyAsync(back, ob, 2 * b_maps + b_npe + STATUS_BYTES, cudaMemcpyDeviceToHost, st),
           "copy outputs");
    } else {
        CK(h, cudaMemcpyAsync(maps, d_maps, total * sizeof(uint32_t), cudaMemcpyDeviceToHost, st), "copy maps");
        CK(h, cudaMemcpyAsync(tmin, d_keys, total * sizeof(float), cudaMemcpyDeviceToHost, st), "copy tmin");
        CK(h, cudaMemcpyAsync(npe, d_npe, (size_t)n_segments * sizeof(int32_t), cudaMemcpyDeviceToHost, st), "copy npe");
        CK(h, cudaMemcpyAsync(counters, d_ctr, sizeof(cl_counters), cudaMemcpyDeviceToHost, st), "copy counters");
    }
    if (want_rec && n > 0) {
        const size_t m = (size_t)n;
        if (records->status) CK(h, cudaMemcpyAsync(records->status, drec.status, m, cudaMemcpyDeviceToHost, st), "copy status");
        if (records->idx) CK(h, cudaMemcpyAsync(records->idx, drec.idx, 2 * m, cudaMemcpyDeviceToHost, st), "copy idx");
        if (records->t) CK(h, cudaMemcpyAsync(records->t, drec.t, 4 * m, cudaMemcpyDeviceToHost, st), "copy t");
        if (records->bounces) CK(h, cudaMemcpyAsync(records->bounces, drec.bounces, 4 * m, cudaMemcpyDeviceToHost, st), "copy bounces");
    }
    if (!gathered) return collect(h, st);
    CK(h, cudaStreamSynchronize(st), "stream synchronize");
    unsigned long long status[2];
    memcpy(maps, back, total * sizeof(uint32_t));
    memcpy(tmin, back + b_maps, total * sizeof(float));
    memcpy(npe, back + 2 * b_maps, (size_t)n_segments * sizeof(int32_t));
    memcpy(counters, back + 2 * b_maps + b_npe, sizeof(cl_counters));
    memcpy(status, back + 2 * b_maps + b_npe + 8 * N_STATUS, sizeof status);
    return report(h, status[0], (unsigned int)status[1]);
}

int cl_run_segments_device(cl_handle* h, const cl_box* box, const cl_optical_params* op,
                           const cl_readout* ro, const cl_time_binning* tb,
                           const float* d_sx, const float* d_sy, const float* d_sz,
                           const float* d_st, const int64_t* d_src_offsets,
                           const int32_t* d_src_segment, int64_t n_src, int64_t n_segments,
                           int64_t n_photons, uint64_t seed, uint64_t pid_offset,
                           float tau_ns, int32_t max_bounces,
                           uint32_t* d_maps, float* d_tmin, int32_t* d_npe,
                           cl_counters* d_counters, const cl_records* d_records, void* stream)
{
    if (!h) return CL_ERR_STATE;
    h->err[0] = 0;
    int rc = check_params(h, box, op, ro, tb, tau_ns, max_bounces);
    if (rc != CL_OK) return rc;
    if (n_src < 1 || n_segments < 1) return set_err(h, CL_ERR_ARG, "need n_src >= 1 and n_segments >= 1");
    if (!d_sx || !d_sy || !d_sz || !d_src_offsets || !d_src_segment)
        return set_err(h, CL_ERR_ARG, "null source array");
    if (!d_maps || !d_tmin || !d_npe || !d_counters) return set_err(h, CL_ERR_ARG, "null output buffer");
    CK(h, cudaSetDevice(h->device), "cudaSetDevice");
    cudaStream_t st = stream ? (cudaStream_t)stream : h->stream;
    const int64_t n = n_photons;
    if (n < 0) return set_err(h, CL_ERR_ARG, "negative photon total");
    const Physics P = make_physics(box, op, ro, tb, tau_ns, max_bounces, seed);
    return enqueue_segments(h, P, d_sx, d_sy, d_sz, d_st, d_src_offsets, d_src_segment, n_src, n_segments,
                            n, pid_offset, d_maps, (uint32_t*)d_tmin, d_npe,
                            (unsigned long long*)d_counters, d_records, st);
}

int cl_run_segments_moments_device(cl_handle* h, const cl_box* box, const cl_optical_params* op,
                                   const cl_readout* ro, const cl_time_binning* tb,
                                   const float* d_sx, const float* d_sy, const float* d_sz,
                                   const float* d_st, const int64_t* d_src_offsets,
                                   const int32_t* d_src_segment, int64_t n_src, int64_t n_segments,
                                   int64_t n_photons, uint64_t seed, uint64_t pid_offset,
                                   float tau_ns, int32_t max_bounces,
                                   uint32_t* d_maps, float* d_tmin, int32_t* d_npe,
                                   cl_counters* d_counters, uint64_t* d_tsum, uint64_t* d_tsum2,
                                   void* stream)
{
    if (!h) return CL_ERR_STATE;
    h->err[0] = 0;
    int rc = check_params(h, box, op, ro, tb, tau_ns, max_bounces);
    if (rc != CL_OK) return rc;
    if (n_src < 1 || n_segments < 1) return set_err(h, CL_ERR_ARG, "need n_src >= 1 and n_segments >= 1");
    if (!d_sx || !d_sy || !d_sz || !d_src_offsets || !d_src_segment)
        return set_err(h, CL_ERR_ARG, "null source array");
    if (!d_maps || !d_tmin || !d_npe || !d_counters || !d_tsum || !d_tsum2)
        return set_err(h, CL_ERR_ARG, "null output buffer");
    if (n_photons < 0) return set_err(h, CL_ERR_ARG, "negative photon total");
    CK(h, cudaSetDevice(h->device), "cudaSetDevice");
    cudaStream_t st = stream ? (cudaStream_t)stream : h->stream;
    const Physics P = make_physics(box, op, ro, tb, tau_ns, max_bounces, seed);
    return enqueue_segments(h, P, d_sx, d_sy, d_sz, d_st, d_src_offsets, d_src_segment, n_src, n_segments,
                            n_photons, pid_offset, d_maps, (uint32_t*)d_tmin, d_npe,
                            (unsigned long long*)d_counters, nullptr, st,
                            (unsigned long long*)d_tsum, (unsigned long long*)d_tsum2);
}

int cl_run_events_surrogate_device(cl_handle* h, const cl_box* box, const cl_optical_params* op,
                                   const cl_readout* ro, const cl_time_binning* tb,
                                   const float* d_sx, const float* d_sy, const float* d_sz,
                                   const float* d_st, const int64_t* d_src_offsets,
                                   const int32_t* d_src_segment, int64_t n_src, int64_t n_photons,
                                   uint64_t seed, uint64_t pid_offset, float tau_ns, int32_t max_bounces,
                                   const float* d_site_p, const float* d_site_tmean,
                                   const float* d_site_tsig, const uint8_t* d_site_flag,
                                   const float* d_site_t0, const int64_t* d_site_photons,
                                   const int32_t* d_site_segment, int64_t n_sites, uint64_t sample_seed,
                                   int64_t n_segments, uint32_t* d_maps, float* d_tmin, int32_t* d_npe,
                                   cl_counters* d_counters, uint64_t* d_sampled, void* stream)
{
    if (!h) return CL_ERR_STATE;
    h->err[0] = 0;
    int rc = check_params(h, box, op, ro, tb, tau_ns, max_bounces);
    if (rc != CL_OK) return rc;
    if (n_segments < 1) return set_err(h, CL_ERR_ARG, "need n_segments >= 1");
    if (n_src < 0 || n_sites < 0 || n_photons < 0) return set_err(h, CL_ERR_ARG, "negative size");
    if (n_src == 0 && n_photons != 0) return set_err(h, CL_ERR_ARG, "photons without Monte Carlo sources");
    if (n_src > 0 && (!d_sx || !d_sy || !d_sz || !d_src_offsets || !d_src_segment))
        return set_err(h, CL_ERR_ARG, "null source array");
    if (n_sites > 0 && (!d_site_p || !d_site_tmean || !d_site_tsig || !d_site_t0 || !d_site_photons ||
                        !d_site_segment))
        return set_err(h, CL_ERR_ARG, "null surrogate site array");
    if (!d_maps || !d_tmin || !d_npe || !d_counters) return set_err(h, CL_ERR_ARG, "null output buffer");
    CK(h, cudaSetDevice(h->device), "cudaSetDevice");
    cudaStream_t st = stream ? (cudaStream_t)stream : h->stream;
    SurSampleArgs sa;
    memset(&sa, 0, sizeof sa);
    sa.p = d_site_p; sa.tmean = d_site_tmean; sa.tsig = d_site_tsig; sa.flag = d_site_flag;
    sa.t0 = d_site_t0; sa.photons = d_site_photons; sa.seg = d_site_segment; sa.n = n_sites;
    sa.n_seg = n_segments;
    sa.cells = ro->grid.nx * ro->grid.ny;
    sa.k0 = (uint32_t)sample_seed; sa.k1 = (uint32_t)(sample_seed >> 32);
    sa.tau = tau_ns;
    sa.stats = (unsigned long long*)d_sampled;
    if (d_sampled) CK(h, cudaMemsetAsync(d_sampled, 0, 2 * sizeof(uint64_t), st), "zero sampler stats");
    const Physics P = make_physics(box, op, ro, tb, tau_ns, max_bounces, seed);
    return enqueue_segments(h, P, d_sx, d_sy, d_sz, d_st, d_src_offsets, d_src_segment, n_src, n_segments,
                            n_photons, pid_offset, d_maps, (uint32_t*)d_tmin, d_npe,
                            (unsigned long long*)d_counters, nullptr, st, nullptr, nullptr, &sa);
}

int cl_sync(cl_handle* h, void* stream)
{
    if (!h) return CL_ERR_STATE;
    CK(h, cudaSetDevice(h->device), "cudaSetDevice");
    return collect(h, stream ? (cudaStream_t)stream : h->stream);
}

int cl_debug_eval(cl_handle* h, int fn, const void* in, void* out, int64_t n, uint64_t seed, int32_t n_per)
{
    if (!h) return CL_ERR_STATE;
    h->err[0] = 0;
    if (n < 0 || !out || (fn != 4 && fn != 6 && !in)) return set_err(h, CL_ERR_ARG, "bad debug arguments");
    if (fn < 0 || fn > 12) return set_err(h, CL_ERR_ARG, "unknown debug function");
    if (fn == 4 && n_per < 1) return set_err(h, CL_ERR_ARG, "n_per must be >= 1");
    CK(h, cudaSetDevice(h->device), "cudaSetDevice");
    cudaStream_t st = h->stream;
    if (fn == 6) {
        // the handle's table of the logs of the uniforms (2^24 floats)
        if (!h->logtab.p) return set_err(h, CL_ERR_STATE, "this handle has no log table");
        if (n > (1 << 24)) return set_err(h, CL_ERR_ARG, "the log table has 2^24 entries");
        CK(h, cudaMemcpyAsync(out, h->logtab.p, 4 * (size_t)n, cudaMemcpyDeviceToHost, st), "copy table");
        CK(h, cudaStreamSynchronize(st), "stream synchronize");
        return CL_OK;
    }
    size_t in_b = 0, out_b = 0;
    if (fn <= 2) { in_b = 4 * (size_t)n; out_b = 4 * (size_t)n; }
    else if (fn == 3 || fn == 5) { in_b = 16 * (size_t)n; out_b = 16 * (size_t)n; }
    else if (fn >= 7) {
        constexpr size_t ni[6] = {1, 1, 9, 4, 3, 9}, no[6] = {1, 1, 4, 2, 2, 3};
        in_b = 4 * ni[fn - 7] * (size_t)n;
        out_b = 4 * no[fn - 7] * (size_t)n;
    }
    else { out_b = 4 * (size_t)n * (size_t)n_per; }
    int rc = ensure(h, h->dbg, align256(in_b) + align256(out_b) + 256);
    if (rc != CL_OK) return rc;
    char* din = (char*)h->dbg.p;
    char* dout = din + align256(in_b);
    if (in_b) CK(h, cudaMemcpyAsync(din, in, in_b, cudaMemcpyHostToDevice, st), "copy in");
    const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 148 * 16));
    const uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
    if (n > 0) {
        if (fn <= 2) debug_math_kernel<<<grid, 256, 0, st>>>(fn, (const float*)din, (float*)dout, n);
        else if (fn == 3 || fn == 5)
            debug_philox_kernel<<<grid, 256, 0, st>>>(fn == 5, (const uint32_t*)din, (uint32_t*)dout, n, k0, k1);
        else if (fn >= 7) debug_step_kernel<<<grid, 256, 0, st>>>(fn, (const float*)din, (float*)dout, n);
        else debug_randu_kernel<<<grid, 256, 0, st>>>((float*)dout, n, n_per, k0, k1);
        CK(h, cudaGetLastError(), "debug kernel launch");
    }
    if (out_b) CK(h, cudaMemcpyAsync(out, dout, out_b, cudaMemcpyDeviceToHost, st), "copy out");
    CK(h, cudaStreamSynchronize(st), "stream synchronize");
    return CL_OK;
}

}  // extern "C"

// ===========================================================================
// Allocation-free entry point (cl_run_photons_noalloc).
//
// For callers that cannot let a library call cudaMalloc (device memory owned
// by a pool/caching allocator or a fixed budget; loops where cudaMalloc or
// cudaFree would synchronise the device).  All device memory it touches is
// the file-scope array below, CL_NOALLOC_SCRATCH_BYTES long, which each GPU
// that loads this library holds until the process exits.  Every call reuses
// (and overwrites) the whole array: calls that overlap on the GPU race.
// ===========================================================================
static __device__ __align__(256) unsigned char g_noalloc_scratch[CL_NOALLOC_SCRATCH_BYTES];

namespace {
constexpr int NOALLOC_MAX_DEVICES = 64;
std::mutex g_noalloc_mu;
struct NoallocDevice {
    bool ready = false;
    unsigned char* base = nullptr;   // device address of g_noalloc_scratch on this device
    int num_sms = 0;
    int max_smem_optin = 0;
    int max_smem_per_sm = 0;
};
NoallocDevice g_noalloc_dev[NOALLOC_MAX_DEVICES];

// Once per device, with that device current: look up the array's device
// address (host code cannot use the symbol itself as a device pointer) and
// the launch limits.  Allocates nothing.
int noalloc_setup(int dev, NoallocDevice** out)
{
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    NoallocDevice& d = g_noalloc_dev[dev];
    if (!d.ready) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&d.num_sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess)
            e = cudaDeviceGetAttribute(&d.max_smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        if (e == cudaSuccess)
            e = cudaDeviceGetAttribute(&d.max_smem_per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
        if (e != cudaSuccess) {
            cudaGetLastError();
            snprintf(g_create_err, sizeof g_create_err, "cl_run_photons_noalloc: set-up on device %d: %s",
                     dev, cudaGetErrorString(e));
            return CL_ERR_CUDA;
        }
        set_kernel_attrs<POINT, false, true>(d.max_smem_optin, false);
        set_kernel_attrs<POINT, false, false>(d.max_smem_optin, false);
        cudaGetLastError();
        d.base = (unsigned char*)p;
        d.ready = true;
    }
    *out = &d;
    return CL_OK;
}
}  // namespace

extern "C" int cl_run_photons_noalloc(const cl_box* box, const cl_optical_params* op,
                                      const cl_readout* ro, const cl_time_binning* tb,
                                      const float* px, const float* py, const float* pz,
                                      const float* pt, int32_t npos,
                                      int64_t n_photons, uint64_t seed, uint64_t pid_offset,
                                      float tau_ns, int32_t max_bounces,
                                      uint32_t* counts, float* first_ns, cl_counters* counters,
                                      void* stream)
{
    g_create_err[0] = 0;
    // A stack handle carries the launch settings and collects error messages;
    // its scratch words point into the static array.  Nothing is allocated.
    cl_handle tmp;
    auto fail = [&](int rc) {
        snprintf(g_create_err, sizeof g_create_err, "cl_run_photons_noalloc: %s", tmp.err);
        return rc;
    };
    int rc = check_params(&tmp, box, op, ro, tb, tau_ns, max_bounces);
    if (rc != CL_OK) return fail(rc);
    if (npos < 1 || !px || !py || !pz) return fail(set_err(&tmp, CL_ERR_ARG, "need npos >= 1 source positions"));
    if (n_photons < 0) return fail(set_err(&tmp, CL_ERR_ARG, "n_photons must be >= 0"));
    if (!counts || !first_ns || !counters) return fail(set_err(&tmp, CL_ERR_ARG, "null output buffer"));

    const int cells = ro->grid.nx * ro->grid.ny;
    const size_t n_counts = (size_t)cells * (size_t)(tb->nbins + 1);
    const size_t b_words = 256, b_ctr = 256;
    const size_t b_counts = align256(n_counts * sizeof(uint32_t));
    const size_t b_keys = align256((size_t)cells * sizeof(uint32_t));
    const size_t b_src = align256((size_t)npos * sizeof(float));
    const size_t need = b_words + b_ctr + b_counts + b_keys + 4 * b_src;
    if (need > (size_t)CL_NOALLOC_SCRATCH_BYTES)
        return fail(set_err(&tmp, CL_ERR_ARG,
                            "staged data needs %zu bytes (npos %d, %d cells x %d bins) but the "
                            "static device array holds %u bytes",
                            need, (int)npos, cells, tb->nbins + 1, (unsigned)CL_NOALLOC_SCRATCH_BYTES));

    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES) {
        cudaGetLastError();
        return fail(set_err(&tmp, CL_ERR_CUDA, "no current CUDA device (%s)",
                            e != cudaSuccess ? cudaGetErrorString(e) : "device index out of range"));
    }
    NoallocDevice* nd = nullptr;
    if ((rc = noalloc_setup(dev, &nd)) != CL_OK) return rc;

    tmp.device = dev;
    tmp.num_sms = nd->num_sms;
    tmp.max_smem_optin = nd->max_smem_optin;
    tmp.max_smem_per_sm = nd->max_smem_per_sm;
    tmp.scratch.p = nd->base;                 // queue / steps / done / err words
    tmp.scratch.cap = b_words;
    unsigned char* base = nd->base;
    unsigned long long* d_ctr = (unsigned long long*)(base + b_words);
    uint32_t* d_counts = (uint32_t*)(base + b_words + b_ctr);
    uint32_t* d_keys = (uint32_t*)(base + b_words + b_ctr + b_counts);
    float* d_px = (float*)(base + b_words + b_ctr + b_counts + b_keys);
    float* d_py = (float*)((unsigned char*)d_px + b_src);
    float* d_pz = (float*)((unsigned char*)d_py + b_src);
    float* d_pt = (float*)((unsigned char*)d_pz + b_src);
    cudaStream_t st = (cudaStream_t)stream;

#define NK(call, what)                                                        \
    do {                                                                      \
        cudaError_t e_ = (call);                                              \
        if (e_ != cudaSuccess) return fail(cuda_fail(&tmp, e_, (what)));      \
    } while (0)
    NK(cudaMemcpyAsync(d_px, px, npos * sizeof(float), cudaMemcpyHostToDevice, st), "copy px");
    NK(cudaMemcpyAsync(d_py, py, npos * sizeof(float), cudaMemcpyHostToDevice, st), "copy py");
    NK(cudaMemcpyAsync(d_pz, pz, npos * sizeof(float), cudaMemcpyHostToDevice, st), "copy pz");
    if (pt) NK(cudaMemcpyAsync(d_pt, pt, npos * sizeof(float), cudaMemcpyHostToDevice, st), "copy pt");

    // The init kernel clears the counts, keys, counters and queue words left
    // by the previous call before the transport kernel runs.
    const Physics P = make_physics(box, op, ro, tb, tau_ns, max_bounces, seed);
    rc = enqueue_point(&tmp, P, d_px, d_py, d_pz, pt ? d_pt : nullptr, npos, n_photons, pid_offset,
                       d_counts, d_keys, d_ctr, nullptr, st);
    if (rc != CL_OK) return fail(rc);
    NK(cudaMemcpyAsync(counts, d_counts, n_counts * sizeof(uint32_t), cudaMemcpyDeviceToHost, st), "copy counts");
    NK(cudaMemcpyAsync(first_ns, d_keys, (size_t)cells * sizeof(float), cudaMemcpyDeviceToHost, st), "copy first_ns");
    NK(cudaMemcpyAsync(counters, d_ctr, sizeof(cl_counters), cudaMemcpyDeviceToHost, st), "copy counters");
#undef NK
    rc = collect(&tmp, st);
    if (rc != CL_OK) return fail(rc);
    return CL_OK;
}
