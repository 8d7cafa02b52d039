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
