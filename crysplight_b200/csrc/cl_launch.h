// cl_launch.h — grid, block and work-queue chunk of a transport launch (host
// arithmetic alone, so that it can be checked without a GPU).
#pragma once

#include <cstdint>

namespace cl {

constexpr int SPREAD_WARPS = 8;          // warps per SM of a launch of few photons
constexpr int AUTO_THREADS = 256;        // threads per CTA where none are asked for
constexpr int SPREAD_THREADS = 128;      // and of a launch of few photons
constexpr int CHUNKS_PER_WARP = 16;      // queue chunks a resident warp gets at least
constexpr int MAX_WARP_CHUNK = 256;

// What cl_set_launch asked for (0: automatic).
struct LaunchSetting {
    int ctas_per_sm = 0, threads = 0, warp_chunk = 0;
};
struct LaunchShape {
    int64_t grid;
    int threads;
    int32_t warp_chunk;
};

// Shape for n photons where `resident` CTAs of setting.threads (or AUTO_THREADS)
// threads fit on an SM.  What was asked for is kept; the rest follows n.
inline LaunchShape launch_shape(int64_t n, int num_sms, int resident, const LaunchSetting& set)
{
    int per_sm = resident;
    if (set.ctas_per_sm > 0 && set.ctas_per_sm < per_sm) per_sm = set.ctas_per_sm;
    int threads = set.threads > 0 ? set.threads : AUTO_THREADS;
    int64_t grid = (int64_t)num_sms * per_sm;
    int64_t chunk = set.warp_chunk;
    if (chunk <= 0) {
        // automatic: the largest chunk (fewest queue atomics) that still gives
        // every resident warp about CHUNKS_PER_WARP chunks, so the end of the
        // queue stays balanced; between 32 and MAX_WARP_CHUNK photons
        const int64_t warps = grid * (threads / 32);
        chunk = n / (warps * CHUNKS_PER_WARP);
        chunk = (chunk < 32 ? 32 : (chunk > MAX_WARP_CHUNK ? MAX_WARP_CHUNK : chunk)) & ~(int64_t)31;
        // fewer photons than two warps per scheduler hold: spread them over that
        // many warps (or the resident ones), some lanes each.  The time is the
        // longest photon's chain of steps, and a warp with few lanes runs fewer of
        // a step's branches: CsI(Tl) 2,000 photons 271 -> 245 us, 20,000 294 -> 285
        // us, BGO 500 photons 946 -> 849 us; with 4 warps per SM 8,000 photons take
        // 262 us instead of 257, with 16 269 us
        int64_t spread = (int64_t)num_sms * SPREAD_WARPS;
        if (warps < spread) spread = warps;
        if (n < spread * 32) {
            chunk = (n + spread - 1) / spread;
            if (set.threads <= 0 && set.ctas_per_sm <= 0) threads = SPREAD_THREADS;
        }
    }
    // no more CTAs than warps' worth of first chunks
    const int64_t warps_needed = (n + chunk - 1) / chunk;
    const int64_t ctas_needed = (warps_needed + (threads / 32) - 1) / (threads / 32);
    if (grid > ctas_needed) grid = ctas_needed > 0 ? ctas_needed : 1;
    return LaunchShape{grid, threads, (int32_t)chunk};
}

}  // namespace cl
