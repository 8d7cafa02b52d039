// Pixels handed to the lanes of a warp, and rows counted as they complete:
// the work split of the escape-time kernels.
//
// A warp pulls tiles of 32 pixels (8x4 of the frame, or 32 entries of a
// list) and keeps the current one in shared memory.  A lane whose pixel is
// done takes the tile's next pixel, so lanes do not wait for the slowest
// pixel of a tile: around a boundary point, where neighbours' counts differ
// by thousands of iterations, whole tiles left nearly half of the lanes idle.
#pragma once

#include "internal.h"

namespace mdz {

constexpr int kTileW = 8;
constexpr int kTileH = 4;

// The warp's current tile: `count` pixels, `left` of them not taken yet.
struct TileFeed {
    int count = 0, left = 0;
    bool more = true;    // tiles may be left
    bool first = true;   // no tile pulled yet
};

// Number of the warp's next tile (on every lane), or ~0u when stopped.  The
// first one is dealt out, block by block and then warp by warp, so that a
// launch of few tiles spreads over the SMs and their schedulers (pulled from
// the counter, the 41 tiles of a list went to the warps of a few SMs: 26 to
// 33 ms where 41 SMs take 12); later ones come from the counter.
__device__ __forceinline__ unsigned next_tile(TileFeed& f, unsigned* counter, volatile int* stop)
{
    unsigned t = ~0u;
    const unsigned warps = blockDim.x >> 5;
    if ((threadIdx.x & 31) == 0 && !(stop && *stop))
        t = f.first ? (threadIdx.x >> 5) * gridDim.x + blockIdx.x
                    : warps * gridDim.x + atomicAdd(counter, 1u);
    f.first = false;
    return __shfl_sync(0xffffffffu, t, 0);
}

// Gives pixels to the lanes with `idle` set.  next() returns, on every lane,
// the next tile's number or ~0u; pixel(tile, px, row) sets the lane's pixel of
// that tile and says whether it is in the frame; stash(k, px, row) keeps it as
// the tile's k-th; take(k) starts the lane on the k-th.  All lanes call it.
template <class Next, class Pixel, class Stash, class Take>
__device__ __forceinline__ void feed_lanes(TileFeed& f, bool idle, Next next, Pixel pixel,
                                           Stash stash, Take take)
{
    const unsigned below = (1u << (threadIdx.x & 31)) - 1u;
    unsigned want = __ballot_sync(0xffffffffu, idle);
    while (want && (f.left || f.more)) {
        if (!f.left) {
            const unsigned t = next();
            if (t == ~0u) {
                f.more = false;
                break;
            }
            int px = 0, row = 0;
            const bool in = pixel(t, px, row);
            const unsigned m = __ballot_sync(0xffffffffu, in);
            if (in)
                stash(__popc(m & below), px, row);
            f.count = f.left = __popc(m);
            __syncwarp();
        }
        // the k-th idle lane takes the k-th pixel left
        const int k = __popc(want & below);
        const bool takes = idle && ((want >> (threadIdx.x & 31)) & 1u) && k < f.left;
        if (takes)
            take(f.count - f.left + k);
        const unsigned took = __ballot_sync(0xffffffffu, takes);
        f.left -= __popc(took);
        want &= ~took;
    }
}

// The end of a launch.  Once the tiles are used up, lanes go idle one by one
// and a warp of seven pixels costs the pipes as much as one of 32: the warps
// of a block then move their pixels together whenever these fit in fewer
// warps.  A warp that has found no tile sets `dry` (the others then need not
// ask for one); each one, at its next look(), publishes how many pixels it
// holds, and calls merge() when a warp can be saved or when it has no pixel
// itself.
template <int WARPS>
struct LaneMerge {
    int held[WARPS];   // at most this many pixels in the warp
    int now[WARPS];    // merge(): its pixels, and those of its tile left (<< 16)
    int dry;

    __device__ __forceinline__ void init()
    {
        if (threadIdx.x < WARPS)
            held[threadIdx.x] = 64;
        if (threadIdx.x == 0)
            dry = 0;
        __syncthreads();
    }
    __device__ __forceinline__ void set_dry() { *(volatile int*)&dry = 1; }
    __device__ __forceinline__ bool is_dry()
    {
        return __any_sync(0xffffffffu, *(volatile int*)&dry != 0);
    }

    // Publishes the warp's pixels; whether it is to call merge().  (Until its
    // first look a warp counts as 64, more than it can hold, so the sum only
    // falls: once one warp has gone to merge(), all follow at their next look.)
    __device__ __forceinline__ bool look(const TileFeed& f, bool active, int kept)
    {
        const int lane = threadIdx.x & 31;
        const int n = __popc(__ballot_sync(0xffffffffu, active));
        if (lane == 0)
            *(volatile int*)&held[threadIdx.x >> 5] = n + f.left;
        __syncwarp();
        const int all = __reduce_add_sync(
            0xffffffffu, lane < WARPS ? *(volatile int*)&held[lane] : 0);
        return n == 0 || (all + 31) / 32 < kept;
    }

    // All warps of the block: moves the pixels of warps `kept` and up (set
    // here: as few as hold them all; warp w is scheduler w mod 4's, so the
    // first ones share the schedulers evenly) to idle lanes below.  put(k)
    // stores the lane's pixel as the k-th of `cap` in shared memory, get(k)
    // takes it.  False when the block holds no pixel.
    template <class Put, class Get>
    __device__ __forceinline__ bool merge(const TileFeed& f, bool& active, int& kept, int cap,
                                          Put put, Get get)
    {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const unsigned act = __ballot_sync(0xffffffffu, active);
        if (lane == 0)
            now[warp] = __popc(act) | (f.left << 16);
        __syncthreads();
        const int h = lane < WARPS ? now[lane] : 0;
        const int all = __reduce_add_sync(0xffffffffu, h);
        if (!all)
            return false;
        const int n = h & 0xffff;
        kept = ((all & 0xffff) + 31) / 32;
        // pixels to move before warp `lane`'s, or free lanes before its own
        int sum = lane < kept ? 32 - n : n;
        int before = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, before, o);
            if (lane >= o)
                before += v;
        }
        __syncthreads();
        const int total = __shfl_sync(0xffffffffu, before, 31);
        const int room = kept ? __shfl_sync(0xffffffffu, before, kept - 1) : 0;
        const int moving = total - room;
        before -= sum;
        const bool gives = warp >= kept;
        const unsigned mine = gives ? act : ~act;
        const bool moves = (mine >> lane) & 1u;
        const int k = __shfl_sync(0xffffffffu, before, warp) - (gives ? room : 0)
                      + __popc(mine & ((1u << lane) - 1u));
        for (int from = 0; from < moving; from += cap) {
            const bool now = moves && k >= from && k < min(moving, from + cap);
            if (gives && now) {
                put(k - from);
                active = false;
            }
            __syncthreads();
            if (!gives && now) {
                get(k - from);
                active = true;
            }
            const unsigned left = __ballot_sync(0xffffffffu, active);
            if (lane == 0)
                held[warp] = __popc(left) + f.left;
            __syncthreads();
        }
        return true;
    }
};

// Progressive rows: `band` is the 4-row band of a pixel this lane finished
// since the last call, or -1.  The band whose last pixel this was gets its
// host-visible flag (lines_rendered[] + lines_rendered_cond of
// src/render_threads.c).  All lanes call it, after their counts are stored.
__device__ __forceinline__ void count_bands(int W, int nrows, unsigned* done_per_band,
                                            volatile int* flags, int& band)
{
    const bool fin = band >= 0;
    if (!__any_sync(0xffffffffu, fin))
        return;
    if (flags)
        __threadfence_system();
    __syncwarp();
    const unsigned grp = __match_any_sync(0xffffffffu, band);
    if (fin && (int)(threadIdx.x & 31) == __ffs(grp) - 1) {
        const unsigned n = (unsigned)__popc(grp);
        const unsigned rows = min((unsigned)kTileH, (unsigned)(nrows - band * kTileH));
        const unsigned done = atomicAdd(done_per_band + band, n) + n;
        if (done == rows * (unsigned)W && flags) {
            __threadfence_system();
            flags[band] = 1;
        }
    }
    band = -1;
}

}  // namespace mdz
