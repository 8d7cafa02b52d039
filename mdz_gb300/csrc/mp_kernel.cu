// Multi-limb fixed-point escape-time kernel: the GPU form of MDZ's
// multiprecision path.
//
// Reference loops (per iteration, same operation order):
//   Mandelbrot          src/frac_mandel.c:25-52        (MPFR)  :55-82  (GMP)
//   burning ship        src/frac_burning_ship.c:27-55  (MPFR)  :58-86  (GMP)
//   generalized celtic  src/frac_generalized_celtic.c:27-55    :58-86
//   hybrid              src/frac_variant.c:26-55               :58-87
//   pixel -> coordinate src/fractal.c:159-192 (MPFR), :299-332 (GMP)
// MPFR/GMP floats are replaced by N-word fixed point (fixed_point.cuh) with
// at least precision+8 bits; counts agree with MPFR at the same precision
// wherever MPFR at twice the precision agrees with it.
//
// One thread iterates one pixel; magnitudes and sign masks are kept
// separately so the three products per iteration run on magnitudes.  c stays
// in registers up to 16 words and moves to shared memory above that so the
// 34/36-word (1088-bit class) kernels fit in registers.  Warps pull 8x4 tiles
// (or 32 entries of a list) from an atomic counter, and a lane takes a new
// pixel once kRefill lanes are idle (pixel_feed.cuh).
//
// What bounds it is the integer multiplier: N = 10 takes 126 partial products
// an iteration at 1.1 cycles of an SM each, N = 34 1272 (fixed_point.cuh).
#include <algorithm>
#include <type_traits>

#include "fixed_point.cuh"
#include "internal.h"
#include "pixel_feed.cuh"
#include "serve.h"

namespace mdz {
namespace {

constexpr int kRefill = 4;        // idle lanes that make a warp take new pixels
constexpr int kRefillEvery = 8;   // iterations between looks at the idle lanes
constexpr int kLookEvery = 8;     // these between looks at the block's other warps

template <int N>
struct CRegs {
    uint32_t w[N];
    __device__ __forceinline__ uint32_t operator()(int k) const { return w[k]; }
    __device__ __forceinline__ void set(int k, uint32_t v) { w[k] = v; }
};

template <int N>
struct CShared {
    uint32_t* base;  // word k of this thread at base[k * stride]
    int stride;
    __device__ __forceinline__ uint32_t operator()(int k) const { return base[k * stride]; }
    __device__ __forceinline__ void set(int k, uint32_t v) { base[k * stride] = v; }
};

// Top two words of a fixed-point number as a float (value < 128 in size).
template <int N>
__device__ __forceinline__ float fx_top_float(const uint32_t (&x)[N])
{
    return (float)(int32_t)x[N - 1] * 5.9604645e-8f /* 2^-24 */
           + (float)x[N - 2] * 1.3877788e-17f /* 2^-56 */;
}

// Whether a pixel's |z|^2 is formed when it is done, from the squares' top words
// (four registers), and not in the step that ends it: the step then has no
// branch for it.  3000 iterations of one pixel at 4 words 0.73 ms and 0.80 (the
// kernel before MpOrbit 0.71), 80 and 256 bits, 320x240, 6.9 and 18.0 ms and 7.2 and
// 18.9; from 16 to 34 words 3% to 1%.  At 36 words the registers do not go round:
// 1088 bits 67.7 ms and 64.9.
template <int N>
constexpr bool late_mag()
{
    return N <= 34;
}

// A pixel's orbit between iterations: |wre|, |wim| with their sign masks and
// wre^2 - wim^2, after `wz` iterations.
template <int N>
struct MpOrbit {
    uint32_t wre[N], wim[N], d[N];
    uint32_t sre, sim;
    uint32_t wz;
    uint32_t top[late_mag<N>() ? 4 : 1];   // of wim^2 and of wre^2, high word first
};

// The squares of |wre|, |wim|: sets d (and top); returns whether |z|^2 > 4, and
// else |z|^2 (rounded) when it is or when `want_mag`.
template <int N>
__device__ __forceinline__ bool mp_squares(MpOrbit<N>& o, bool want_mag, float& mag)
{
    uint32_t acc[N + 2], wre2[N], wim2[N];
    fx::sqr_trunc<N>(o.wim, acc);
    fx::extract<N, 24>(acc, wim2);
    fx::sqr_trunc<N>(o.wre, acc);
    fx::extract<N, 24>(acc, wre2);
    const bool escaped = fx::sum_gt4<N>(wim2, wre2);
    if constexpr (late_mag<N>()) {
        o.top[0] = wim2[N - 1];
        o.top[1] = wim2[N - 2];
        o.top[2] = wre2[N - 1];
        o.top[3] = wre2[N - 2];
    } else if (escaped || want_mag) {
        mag = fx_top_float<N>(wim2) + fx_top_float<N>(wre2);
    }
    fx::sub<N>(wre2, wim2, o.d);
    return escaped;
}

// Signs and magnitudes of a start value in wre, wim.
template <int N>
__device__ __forceinline__ void mp_start(MpOrbit<N>& o)
{
    float mag;
    o.sre = fx::abs_inplace<N>(o.wre);
    o.sim = fx::abs_inplace<N>(o.wim);
    o.wz = 0;
    mp_squares<N>(o, false, mag);   // z_0 = c is not tested
}

// |z|^2 of a z whose square the format may not hold (signed wre, wim).
template <int N>
__device__ __forceinline__ float mp_far_mag(const MpOrbit<N>& o)
{
    const float a = fx_top_float<N>(o.wre), b = fx_top_float<N>(o.wim);
    return a * a + b * b;
}

// The next iteration.  Returns true when z escaped; mag as mp_squares.
// `fold_im`: burning ship; `fold_re`: celtic; `fold_odd`: the hybrid's fold
// on odd iterations.
template <int N, class CG>
__device__ __forceinline__ bool mp_step(MpOrbit<N>& o, const CG& c_re, const CG& c_im, bool fold_im,
                                        bool fold_re, bool fold_odd, bool want_mag, float& mag)
{
    uint32_t acc[N + 2], t[N];
    ++o.wz;
    // wim = 2.0 * wre * wim + c_im   (burning ship: 2 |wre wim| + c_im)
    fx::mul_trunc<N>(o.wre, o.wim, acc);
    fx::extract<N, 23>(acc, t);
    fx::add_signed<N>(c_im, t, fold_im ? 0u : (o.sre ^ o.sim), o.wim);
    // wre = wre2 - wim2 + c_re       (celtic: |wre2 - wim2| + c_re)
    const uint32_t md = (fold_re || (fold_odd && (o.wz & 1u)))
                            ? (uint32_t)((int32_t)o.d[N - 1] >> 31)
                            : 0u;
    fx::add_signed<N>(c_re, o.d, md, o.wre);
    if (fx::big<N>(o.wre) || fx::big<N>(o.wim)) {
        if constexpr (!late_mag<N>())
            mag = mp_far_mag<N>(o);
        return true;
    }
    o.sre = fx::abs_inplace<N>(o.wre);
    o.sim = fx::abs_inplace<N>(o.wim);
    return mp_squares<N>(o, want_mag, mag);
}

// |z|^2 of a finished pixel; mag as its last step left it.
template <int N>
__device__ __forceinline__ float mp_mag(const MpOrbit<N>& o, float mag)
{
    if constexpr (late_mag<N>()) {
        if (fx::big<N>(o.wre) || fx::big<N>(o.wim))
            return mp_far_mag<N>(o);
        const uint32_t im[2] = {o.top[1], o.top[0]}, re[2] = {o.top[3], o.top[2]};
        return fx_top_float<2>(im) + fx_top_float<2>(re);
    }
    return mag;
}

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

template <int N>
__host__ __device__ constexpr bool c_in_smem()
{
    return N > 16;
}

// Threads of a serving block.
template <int N>
__host__ __device__ constexpr int block_threads()
{
    return N > 16 ? 128 : 256;
}

// A frame launch takes one block an SM, whose warps merge as pixels finish
// (pixel_feed.cuh): 320x240 at 80 bits, counts 0.70 of the depth on average,
// 8.08 ms in four blocks of four warps an SM, 6.8 in one of 16.  16 warps hide the
// multiplier's latency best as long as the registers go round, up to 16 words
// (128 a thread, a few spilled): 640x480 to depth 500, all pixels to the end, in
// 16, 12 and 8 warps 4.27, 4.68, 4.74 ms at 10 words, 5.40, 6.02, 5.89 at 12, 7.88,
// 8.81, 8.35 at 16.  At 20 words 12 warps (11.4 ms, 11.5 with 8), above 8: 24 words
// 15.6 ms and 14.7 in 12, but 320x240 to depth 1000 7.85 and 8.93.  (Taken with
// |z|^2 formed in the step; see late_mag.)
template <int N>
__host__ __device__ constexpr int frame_block()
{
    return N > 20 ? 256 : N > 16 ? 384 : 512;
}
constexpr int kFrameMove = 64;   // pixels moved to other warps at a time

template <int N, int FRACTAL, bool JULIA>
__global__ void __launch_bounds__(frame_block<N>(), 1) mp_frame_kernel(MpLaunch p)
{
    extern __shared__ uint32_t smem[];
    constexpr int kBlock = frame_block<N>(), kWarps = kBlock / 32;
    __shared__ int2 tile[kWarps][32];   // the warp's current tile
    __shared__ LaneMerge<kWarps> merge;
    __shared__ uint32_t moved[2 * N + 5][kFrameMove];
    merge.init();
    int kept = kWarps;
    bool dry = false;   // the tiles are used up
    using CGet = typename std::conditional<c_in_smem<N>(), CShared<N>, CRegs<N>>::type;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tiles_x = (p.W + kTileW - 1) / kTileW;
    const int tiles_y = (p.nrows + kTileH - 1) / kTileH;
    const unsigned list_n = p.list ? *p.list_count : 0u;
    const unsigned listed = (list_n + 31u) / 32u;
    // (a short list is mp_split_kernel's or mp_pixel_kernel's)
    const unsigned total = p.list ? (list_n <= p.split_limit ? 0u : listed)
                                  : (unsigned)tiles_x * (unsigned)tiles_y;
    unsigned long long its = 0;
    TileFeed feed;
    bool active = false;   // this lane iterates a pixel
    int ix = 0, lrow = 0;
    int band = -1;
    MpOrbit<N> o;
    CGet c_re, c_im;
    if constexpr (c_in_smem<N>()) {
        c_re = CGet{smem + threadIdx.x, kBlock};
        c_im = CGet{smem + N * kBlock + threadIdx.x, kBlock};
    }
    for (;;) {
        if (p.tile_rows_done && !p.list)
            count_bands(p.W, p.nrows, p.tile_rows_done, p.band_flags, band);
        bool came = false;   // from another warp
        if (dry && merge.look(feed, active, kept)
            && !merge.merge(
                feed, active, kept, kFrameMove,
                [&](int k) {
#pragma unroll
                    for (int j = 0; j < N; ++j) {
                        moved[j][k] = o.wre[j];
                        moved[N + j][k] = o.wim[j];
                    }
                    moved[2 * N][k] = o.sre;
                    moved[2 * N + 1][k] = o.sim;
                    moved[2 * N + 2][k] = o.wz;
                    moved[2 * N + 3][k] = (uint32_t)ix;
                    moved[2 * N + 4][k] = (uint32_t)lrow;
                },
                [&](int k) {
#pragma unroll
                    for (int j = 0; j < N; ++j) {
                        o.wre[j] = moved[j][k];
                        o.wim[j] = moved[N + j][k];
                    }
                    o.sre = moved[2 * N][k];
                    o.sim = moved[2 * N + 1][k];
                    o.wz = moved[2 * N + 2][k];
                    ix = (int)moved[2 * N + 3][k];
                    lrow = (int)moved[2 * N + 4][k];
                    came = true;
                }))
            break;
        bool fresh = false;
        feed_lanes(
            feed, !active,
            [&]() {
                const unsigned n = next_tile(feed, &p.sync->tile_counter, p.stop);
                return n < p.tile_limit && p.tile_base + n < total ? p.tile_base + n : ~0u;
            },
            [&](unsigned t, int& px, int& row) {
                if (p.list) {
                    const unsigned i = t * 32u + lane;
                    const unsigned pix = i < list_n ? p.list[i] : 0u;
                    row = (int)(pix / (unsigned)p.W);
                    px = (int)(pix - (unsigned)row * (unsigned)p.W);
                    return i < list_n;
                }
                const int ty = (int)(t / (unsigned)tiles_x);
                px = (int)(t - (unsigned)ty * (unsigned)tiles_x) * kTileW + (lane & (kTileW - 1));
                row = ty * kTileH + lane / kTileW;
                return px < p.W && row < p.nrows;
            },
            [&](int k, int px, int row) { tile[warp][k] = make_int2(px, row); },
            [&](int k) {
                ix = tile[warp][k].x;
                lrow = tile[warp][k].y;
                fresh = true;
            });
        if (fresh || came) {
            const uint32_t* xs = p.xs + (size_t)ix * N;
            const uint32_t* ys = p.ys + (size_t)lrow * N;
#pragma unroll
            for (int k = 0; k < N; ++k) {
                const uint32_t x = xs[k], y = ys[k];
                if (fresh) {
                    o.wre[k] = x;
                    o.wim[k] = y;
                }
                c_re.set(k, JULIA ? p.julia[k] : x);
                c_im.set(k, JULIA ? p.julia[N + k] : y);
            }
            if (fresh) {
                o.sre = fx::abs_inplace<N>(o.wre);
                o.sim = fx::abs_inplace<N>(o.wim);
                o.wz = 0;
            }
            float mag;
            mp_squares<N>(o, false, mag);   // z_0 = c is not tested
            active = true;
        }
        if (!feed.left && !feed.more && !dry) {
            dry = true;
            if (lane == 0)
                merge.set_dry();
        }
        if (!__any_sync(0xffffffffu, active))
            continue;
        // iterate until enough lanes are idle to be worth a look
        const int enough = (feed.left || feed.more) ? kRefill : 32;
        int looks = kLookEvery;
        do {
            if (active) {
                int u = kRefillEvery;
                bool escaped, done;
                float mag = 0.f;
#pragma unroll 1
                do {
                    escaped = mp_step<N>(o, c_re, c_im, FRACTAL == MDZ_BURNING_SHIP,
                                         FRACTAL == MDZ_GENERALIZED_CELTIC, FRACTAL == MDZ_VARIANT,
                                         o.wz + 1u >= p.depth, mag);
                    done = escaped || o.wz >= p.depth;
                } while (!done && --u);
                if (done) {
                    const uint32_t n = escaped ? o.wz : 0u;
                    const size_t at = (size_t)lrow * p.W + ix;
                    p.out[at] = (int32_t)n;
                    if (p.mag)
                        p.mag[at] = mp_mag<N>(o, mag);
                    its += n ? n : p.depth;
                    active = false;
                    band = lrow / kTileH;
                }
            }
            if (!dry && merge.is_dry()) {
                dry = true;
                feed.more = false;
                break;
            }
            if (dry && --looks == 0)
                break;
        } while (__popc(__ballot_sync(0xffffffffu, !active)) < enough);
    }
    its = warp_sum_u64(its);
    if (lane == 0 && its)
        atomicAdd(&p.sync->iter_sum, its);
    if (p.done.count)
        done_signal(p.done, (unsigned long long)p.tile_base + p.tile_limit >= listed ? 3 : 1);
}

// ---- short lists: four warps for 32 pixels ----
//
// The perturbation hands a few hundred to a few thousand pixels to the
// multi-limb pass, to run thousands of iterations each; one thread a pixel
// takes 1.2 us an iteration at N = 16 and 4.2 us at N = 34 however few they
// are.  Here lane i of each of a block's four warps works on the same pixel,
// with the same truncated products, so the same counts:
//
//  1. Warps 0 and 1 form the product wre wim, the even rows and the odd ones;
//     warps 2 and 3 the squares of wim and wre: N^2 / 4 multiply-adds each.
//  2. Warp 0 adds the product's halves up to the next wim; warp 3 tests the
//     squares and goes on to the next wre.
//
// A barrier ends each step, and no array is read and written in the same one:
// z and what goes with it are read in 1 and written in 2, the products' parts
// the other way round.
//
// What bounds it is latency: each warp's chain of carries, and two barriers an
// iteration.
constexpr int kSplitBlock = 128;

template <int N>
__global__ void __launch_bounds__(kSplitBlock) mp_split_kernel(MpLaunch p, unsigned sms)
{
    __shared__ uint32_t zim[N][32], zre[N][32];   // |wim|, |wre| of each lane's pixel
    __shared__ uint32_t part[N + 2][32];          // the product's odd rows
    __shared__ uint32_t sq[N][32];                // wim^2
    __shared__ uint32_t sign_re[32];              // sign mask of wre
    __shared__ uint32_t top_im[2][32];            // the two top words of wim, signed
    __shared__ int live;
    const unsigned list_n = *p.list_count;
    // a pixel for every block, then a second one, ...: as few blocks an SM as
    // hold the list
    const unsigned all = sms * ((list_n + 32u * sms - 1u) / (32u * sms));
    const unsigned blocks = all < gridDim.x ? all : gridDim.x;
    if (list_n <= p.pixel_limit || list_n > p.split_limit || blockIdx.x >= blocks
        || blockIdx.x >= list_n)
        return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned at = (unsigned)lane * blocks + blockIdx.x;
    bool done = at >= list_n;
    const unsigned pix = p.list[done ? blockIdx.x : at];
    const bool ship = p.fractal == MDZ_BURNING_SHIP;
    const bool celtic = p.fractal == MDZ_GENERALIZED_CELTIC;
    const bool variant = p.fractal == MDZ_VARIANT;
    uint32_t own[N] = {};   // warp 0: |wim|, warp 3: |wre|
    CRegs<N> c;             // warp 0: c_im, warp 3: c_re
    uint32_t sign = 0, top1 = 0, top0 = 0;
    auto publish = [&](uint32_t (*z)[32]) {
        top1 = own[N - 1];
        top0 = own[N - 2];
        sign = fx::abs_inplace<N>(own);
#pragma unroll
        for (int k = 0; k < N; ++k)
            z[k][lane] = own[k];
        if (warp == 0) {
            top_im[0][lane] = top0;
            top_im[1][lane] = top1;
        } else {
            sign_re[lane] = sign;
        }
    };
    auto start = [&](const uint32_t* z, const uint32_t* julia, uint32_t (*to)[32]) {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            own[k] = z[k];
            c.set(k, p.family == MDZ_FAMILY_JULIA ? julia[k] : own[k]);
        }
        publish(to);
    };
    const unsigned row = pix / (unsigned)p.W;
    if (warp == 0)
        start(p.ys + (size_t)row * N, p.julia + N, zim);
    else if (warp == 3)
        start(p.xs + (size_t)(pix - row * (unsigned)p.W) * N, p.julia, zre);
    auto top_float = [](uint32_t hi, uint32_t lo) {
        return (float)(int32_t)hi * 5.9604645e-8f /* 2^-24 */
               + (float)lo * 1.3877788e-17f /* 2^-56 */;
    };
    auto big = [](uint32_t hi) {
        return (int32_t)hi >= 0x08000000 || (int32_t)hi < -0x08000000;
    };
    unsigned long long its = 0;
    if (threadIdx.x == 0)
        live = 1;
    __syncthreads();
    for (uint32_t wz = 0;; ++wz) {
        uint32_t acc[N + 2], t[N];
        uint32_t sre = 0, im1 = 0, im0 = 0;
        if (warp < 2) {
#pragma unroll
            for (int k = 0; k < N; ++k)
                t[k] = zre[k][lane];
            if (warp == 0) {
                sre = sign_re[lane];
                fx::mul_part<N, 0>(t, own, acc);
            } else {
#pragma unroll
                for (int k = 0; k < N; ++k)
                    own[k] = zim[k][lane];
                fx::mul_part<N, 1>(t, own, acc);
#pragma unroll
                for (int k = 0; k < N + 2; ++k)
                    part[k][lane] = acc[k];
            }
        } else {
            if (warp == 2) {
#pragma unroll
                for (int k = 0; k < N; ++k)
                    own[k] = zim[k][lane];
            } else {
                // before the barrier: past it warp 0 puts the next z's there
                im1 = top_im[1][lane];
                im0 = top_im[0][lane];
            }
            fx::sqr_trunc<N>(own, acc);
            fx::extract<N, 24>(acc, t);
            if (warp == 2) {
#pragma unroll
                for (int k = 0; k < N; ++k)
                    sq[k][lane] = t[k];
            }
        }
        __syncthreads();
        if (warp == 0) {
            // wim = 2.0 * wre * wim + c_im   (burning ship: 2 |wre wim| + c_im)
            fx::add_part<N>(acc, [&](int k) { return part[k][lane]; });
            fx::extract<N, 23>(acc, t);
            fx::add_signed<N>(c, t, ship ? 0u : (sre ^ sign), own);
            publish(zim);
        } else if (warp == 3) {
            uint32_t wim2[N], d[N];
#pragma unroll
            for (int k = 0; k < N; ++k)
                wim2[k] = sq[k][lane];
            if (!done) {
                const bool far = wz && (big(top1) || big(im1));
                const bool over = far || (wz && fx::sum_gt4<N>(wim2, t));   // not z_0 = c
                if (over || wz >= p.depth) {
                    done = true;
                    float mag;
                    if (far) {
                        const float a = top_float(top1, top0), b = top_float(im1, im0);
                        mag = a * a + b * b;
                    } else {
                        mag = fx_top_float<N>(wim2) + fx_top_float<N>(t);
                    }
                    p.out[pix] = over ? (int32_t)wz : 0;
                    if (p.mag)
                        p.mag[pix] = mag;
                    its += over ? wz : p.depth;
                }
            }
            // wre = wre2 - wim2 + c_re       (celtic: |wre2 - wim2| + c_re)
            fx::sub<N>(t, wim2, d);
            const bool fold = celtic || (variant && !(wz & 1u));
            fx::add_signed<N>(c, d, fold ? (uint32_t)((int32_t)d[N - 1] >> 31) : 0u, own);
            const bool any = __any_sync(0xffffffffu, !done);
            if (lane == 0 && !any)
                live = 0;
            publish(zre);
        }
        __syncthreads();
        if (!live)
            break;
    }
    if (warp == 3) {
        its = warp_sum_u64(its);
        if (lane == 0)
            atomicAdd(&p.sync->iter_sum, its);
    }
}

// ---- few pixels, many words: a block a pixel ----
//
// With a few pixels an SM and 24 words or more, a block of 4 (N + 1) threads
// iterates one pixel, with the same truncated products again:
//
//  1. Thread 4 k + s forms one column sum, column N-2+k, in 96 bits: s = 0, 1
//     half of the general product's terms each, s = 2, 3 those of the squares
//     of wim, wre (i < j once, doubled, and the diagonal).
//  2. Two warps, a 64-bit limb a lane, add up the columns: warp 0 the product,
//     and from it the next wim; warp 1 the squares, and from them the escape
//     test and the next wre.  Carries between lanes come from two ballots
//     (generate / propagate, as in mpw_kernel.cu).
//
// What bounds it is latency (two barriers and two warps' chains an iteration)
// for a pixel an SM, issue for more.
template <int N>
__host__ __device__ constexpr int pixel_threads()
{
    return 4 * (N + 1) <= 64 ? 64 : (4 * (N + 1) + 31) / 32 * 32;
}

// x + y + c0 over the warp's limbs, lane 0 lowest.
__device__ __forceinline__ uint64_t warp_add(uint64_t x, uint64_t y, unsigned c0)
{
    const uint64_t s = x + y;
    const unsigned g = __ballot_sync(0xffffffffu, s < x);
    const unsigned p = __ballot_sync(0xffffffffu, s == ~0ull);
    const uint64_t c = ((uint64_t)g + (g | p) + c0) ^ p;
    return s + ((c >> (threadIdx.x & 31)) & 1u);
}

// c + x or, where neg, c - x.
__device__ __forceinline__ uint64_t warp_add_signed(uint64_t c, uint64_t x, bool neg)
{
    return warp_add(c, neg ? ~x : x, neg);
}

template <int N>
__global__ void __launch_bounds__(pixel_threads<N>()) mp_pixel_kernel(MpLaunch p)
{
    constexpr int NL = N / 2;
    constexpr int NC = N + 1;              // columns N-2 .. 2N-2
    __shared__ uint64_t z64[2][NL];        // |wim|, |wre|
    __shared__ uint4 col[3][NC + 3];       // column k at [k + 2]: wre wim, wim^2, wre^2
    __shared__ uint32_t sign[2];           // sign masks of wim, wre
    __shared__ uint64_t top[2];            // signed top limbs of the next wim, wre
    __shared__ int state;                  // 1: done
    __shared__ uint32_t count, next;
    __shared__ float mag;
    const unsigned list_n = *p.list_count;
    if (list_n > p.pixel_limit)
        return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool ship = p.fractal == MDZ_BURNING_SHIP;
    const bool celtic = p.fractal == MDZ_GENERALIZED_CELTIC;
    const bool variant = p.fractal == MDZ_VARIANT;
    // this thread's column sum: terms i0 .. i0 + len - 1
    const int k = tid >> 2, set = tid & 3;
    const int c = N - 2 + k;
    const int ilo = c - (N - 1) > 0 ? c - (N - 1) : 0;
    const int all = (c < N - 1 ? c : N - 1) - ilo + 1;   // terms of the product
    const int i0 = set == 1 ? ilo + (all + 1) / 2 : ilo;
    const int len = k >= NC ? 0 : set == 0 ? (all + 1) / 2 : set == 1 ? all / 2
                                                           : ((c - 1) >> 1) - ilo + 1;
    const int steps = __reduce_max_sync(0xffffffffu, len);
    const uint32_t* zim = (const uint32_t*)z64[0];
    const uint32_t* zre = (const uint32_t*)z64[1];
    const uint32_t* pa = (set == 2 ? zim : zre) + i0;
    const uint32_t* pb = (set == 3 ? zre : zim) + (c - i0);
    // columns that do not exist
    for (int j = tid; j < 9; j += blockDim.x)
        col[j / 3][j % 3 < 2 ? j % 3 : NC + 2] = make_uint4(0u, 0u, 0u, 0u);

    // the sum of a product's columns from word N-2 on, 64 bits a lane
    auto limbs = [&](const uint4* cs) -> uint64_t {
        const bool in = lane <= NL;
        const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
        const uint4 A = in ? cs[2 * lane + 2] : zero, B = in ? cs[2 * lane + 3] : zero;
        const uint4 C = in ? cs[2 * lane] : zero, D = in ? cs[2 * lane + 1] : zero;
        const uint64_t x = (uint64_t)A.y << 32 | A.x, y = (uint64_t)B.x << 32;
        const uint64_t z = (uint64_t)C.z + D.y, w = (uint64_t)D.z << 32;
        uint64_t s = x + y;
        unsigned v = s < x;
        s += z;
        v += s < z;
        s += w;
        v += s < w;
        unsigned from = __shfl_up_sync(0xffffffffu, v, 1);
        if (lane == 0)
            from = 0;
        return warp_add(s, from, 0);
    };
    // that sum's bits from 32 + SH on: floor(P / 2^F) for SH = 24, of 2 P for 23
    auto extract = [&](uint64_t s, int sh) -> uint64_t {
        const uint64_t up = __shfl_down_sync(0xffffffffu, s, 1);
        return lane < NL ? s >> (32 + sh) | up << (32 - sh) : 0ull;
    };
    auto big = [](uint64_t t) {
        const int32_t h = (int32_t)(t >> 32);
        return h >= 0x08000000 || h < -0x08000000;
    };
    auto top_float = [](uint64_t t) {
        return (float)(int32_t)(t >> 32) * 5.9604645e-8f /* 2^-24 */
               + (float)(uint32_t)t * 1.3877788e-17f /* 2^-56 */;
    };
    // |v| to shared memory, its sign mask and signed top limb beside it
    auto publish = [&](uint64_t v, int part) {
        const uint64_t t = __shfl_sync(0xffffffffu, v, NL - 1);
        const bool neg = (int64_t)t < 0;
        if (neg)
            v = warp_add(~v, 0ull, 1);
        if (lane < NL)
            z64[part][lane] = v;
        if (lane == 0) {
            sign[part] = neg ? 0xffffffffu : 0u;
            top[part] = t;
        }
    };
    unsigned long long its = 0;
    for (;;) {
        if (tid == 0) {
            const unsigned t = atomicAdd(&p.sync->tile_counter, 1u);
            next = t < list_n ? p.list[t] : 0xffffffffu;
            state = 0;
        }
        __syncthreads();
        const unsigned pix = next;
        if (pix == 0xffffffffu)
            break;
        // warp 0: y and c_im, warp 1: x and c_re
        uint64_t cst = 0;
        if (warp < 2) {
            const unsigned row = pix / (unsigned)p.W, ix = pix - row * (unsigned)p.W;
            const uint64_t* v = (const uint64_t*)(warp ? p.xs + (size_t)ix * N
                                                       : p.ys + (size_t)row * N);
            const uint64_t z = lane < NL ? v[lane] : 0ull;
            cst = z;
            if (p.family == MDZ_FAMILY_JULIA)
                cst = lane < NL ? ((const uint64_t*)(p.julia + (warp ? 0 : N)))[lane] : 0ull;
            publish(z, warp);
        }
        uint32_t wz = 0;   // iterations done
        for (;;) {
            __syncthreads();
            if (wz && state == 0 && (big(top[0]) || big(top[1]))) {
                if (tid == 0) {
                    const float a = top_float(top[1]), b = top_float(top[0]);
                    mag = a * a + b * b;
                    count = wz;
                }
                break;
            }
            if (state)
                break;
            // column sums
            {
                uint32_t w0 = 0, w1 = 0, w2 = 0;
#pragma unroll 4
                for (int j = 0; j < steps; ++j) {
                    const uint32_t x = j < len ? pa[j] : 0u, y = j < len ? pb[-j] : 0u;
                    asm("mad.lo.cc.u32 %0, %3, %4, %0;\n\t"
                        "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
                        "addc.u32 %2, %2, 0;"
                        : "+r"(w0), "+r"(w1), "+r"(w2) : "r"(x), "r"(y));
                }
                if (set >= 2) {
                    w2 = __funnelshift_l(w1, w2, 1);
                    w1 = __funnelshift_l(w0, w1, 1);
                    w0 <<= 1;
                    const uint32_t h = (k < NC && !(c & 1)) ? (set == 2 ? zim : zre)[c >> 1] : 0u;
                    asm("mad.lo.cc.u32 %0, %3, %3, %0;\n\t"
                        "madc.hi.cc.u32 %1, %3, %3, %1;\n\t"
                        "addc.u32 %2, %2, 0;"
                        : "+r"(w0), "+r"(w1), "+r"(w2) : "r"(h));
                }
                // the product's halves are neighbours
                const uint32_t v0 = __shfl_xor_sync(0xffffffffu, w0, 1);
                const uint32_t v1 = __shfl_xor_sync(0xffffffffu, w1, 1);
                const uint32_t v2 = __shfl_xor_sync(0xffffffffu, w2, 1);
                if (set == 0)
                    asm("add.cc.u32 %0, %0, %3;\n\t"
                        "addc.cc.u32 %1, %1, %4;\n\t"
                        "addc.u32 %2, %2, %5;"
                        : "+r"(w0), "+r"(w1), "+r"(w2) : "r"(v0), "r"(v1), "r"(v2));
                if (k < NC && set != 1)
                    col[set ? set - 1 : 0][k + 2] = make_uint4(w0, w1, w2, 0u);
            }
            const uint32_t sre = sign[1], sim = sign[0];
            __syncthreads();
            ++wz;
            if (warp == 0) {
                // wim = 2.0 * wre * wim + c_im   (burning ship: 2 |wre wim| + c_im)
                const uint64_t t = extract(limbs(col[0]), 23);
                publish(warp_add_signed(cst, t, !ship && sre != sim), 0);
            } else if (warp == 1) {
                const uint64_t wim2 = extract(limbs(col[1]), 24);
                const uint64_t wre2 = extract(limbs(col[2]), 24);
                // |z|^2 > 4 (not of z_0 = c)
                const uint64_t ta = __shfl_sync(0xffffffffu, wim2, NL - 1);
                const uint64_t tb = __shfl_sync(0xffffffffu, wre2, NL - 1);
                const uint32_t sum = (uint32_t)(ta >> 32) + (uint32_t)(tb >> 32);
                bool over = sum > 0x04000000u;
                if (sum - 0x03ffffffu <= 1u) {
                    const uint64_t s = warp_add(wim2, wre2, 0);
                    const uint64_t t = __shfl_sync(0xffffffffu, s, NL - 1);
                    const bool low = __any_sync(0xffffffffu, lane < NL - 1 ? s != 0ull
                                                                           : lane == NL - 1
                                                                                 && (uint32_t)s);
                    over = (uint32_t)(t >> 32) > 0x04000000u
                           || ((uint32_t)(t >> 32) == 0x04000000u && low);
                }
                over = over && wz > 1;
                if (over || wz > p.depth) {
                    if (lane == 0) {
                        state = 1;
                        count = over ? wz - 1 : 0u;
                        mag = top_float(ta) + top_float(tb);
                    }
                } else {
                    // wre = wre2 - wim2 + c_re       (celtic: |wre2 - wim2| + c_re)
                    const uint64_t d = warp_add(wre2, ~wim2, 1);
                    const bool neg = (int64_t)__shfl_sync(0xffffffffu, d, NL - 1) < 0;
                    const bool fold = neg && (celtic || (variant && (wz & 1u)));
                    publish(warp_add_signed(cst, d, fold), 1);
                }
            }
        }
        if (tid == 0) {
            p.out[pix] = (int32_t)count;
            if (p.mag)
                p.mag[pix] = mag;
            its += count ? count : p.depth;
        }
        __syncthreads();
    }
    if (tid == 0 && its)
        atomicAdd(&p.sync->iter_sum, its);
}

// Serving: one step of the multi-limb method over its mixed work queue
// (class `cls`); see serve.h.  State per pixel: |wre| (N words), |wim| (N
// words), the next iteration, the two sign masks.
template <int N>
__global__ void __launch_bounds__(block_threads<N>()) serve_mp_kernel(ServeDev* __restrict__ d,
                                                                     int cls)
{
    extern __shared__ uint32_t smem[];
    if (serve_block_leaves(d, cls))
        return;
    const unsigned cur = d->ctl.cur;
    const unsigned n = d->status.qcount[cls][cur];
    const ServeClassTimer timer(d, cls, cur, n);
    const unsigned* qin = d->queue[cls][cur];
    unsigned* qout = d->queue[cls][cur ^ 1u];
    unsigned* qout_count = &d->status.qcount[cls][cur ^ 1u];
    const unsigned long long cancel = d->ctl.cancel;
    const int lane = threadIdx.x & 31;
    for (;;) {
        unsigned base = 0;
        if (lane == 0)
            base = atomicAdd(&d->qpull[cls], 32u);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= n)
            break;
        const unsigned i = base + lane;
        const bool valid = i < n;
        const unsigned e = valid ? qin[i] : 0u;
        const int slot = (int)(e >> kEntrySlotShift);
        const unsigned pix = e & kEntryPixelMask;
        bool done = false, again = false;
        if (valid) {
            if ((cancel >> slot) & 1ull) {
                done = true;
            } else {
                const ServeReq& rq = d->req[slot];
                const int W = rq.pl.W;
                const int line = (int)(pix / (unsigned)W);
                const int ix = (int)(pix - (unsigned)line * (unsigned)W);
                const uint32_t* xs = rq.xs + (size_t)ix * N;
                const uint32_t* ys = rq.ys + (size_t)line * N;
                // c: the pixel (Mandelbrot family) or the Julia constant
                const uint32_t* cxs = rq.julia ? rq.julia : xs;
                const uint32_t* cys = rq.julia ? rq.julia + N : ys;
                uint32_t* sp = (uint32_t*)(rq.state + (size_t)pix * rq.state_stride);
                MpOrbit<N> o;
                float mag = 0.f;
                if (e & kEntryFresh) {
#pragma unroll
                    for (int k = 0; k < N; ++k) {
                        o.wre[k] = xs[k];
                        o.wim[k] = ys[k];
                    }
                    mp_start<N>(o);
                } else {
#pragma unroll
                    for (int k = 0; k < N; ++k) {
                        o.wre[k] = sp[k];
                        o.wim[k] = sp[N + k];
                    }
                    o.wz = sp[2 * N] - 1u;
                    const uint32_t sg = sp[2 * N + 1];
                    o.sre = (sg & 1u) ? 0xffffffffu : 0u;
                    o.sim = (sg & 2u) ? 0xffffffffu : 0u;
                    mp_squares<N>(o, false, mag);
                }
                const uint32_t depth = rq.pl.depth;
                const uint32_t last = min(o.wz + d->ctl.budget[slot], depth);
                using CGet = typename std::conditional<c_in_smem<N>(), CShared<N>, CRegs<N>>::type;
                CGet c_re, c_im;
                if constexpr (c_in_smem<N>()) {
                    c_re = CGet{smem + threadIdx.x, (int)blockDim.x};
                    c_im = CGet{smem + (size_t)N * blockDim.x + threadIdx.x, (int)blockDim.x};
                }
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    c_re.set(k, cxs[k]);
                    c_im.set(k, cys[k]);
                }
                const int fr = rq.fractal;
                bool escaped = false;
#pragma unroll 1
                while (!escaped && o.wz < last)
                    escaped = mp_step<N>(o, c_re, c_im, fr == MDZ_BURNING_SHIP,
                                         fr == MDZ_GENERALIZED_CELTIC, fr == MDZ_VARIANT,
                                         o.wz + 1u >= depth, mag);
                if (escaped || o.wz >= depth) {
                    rq.pl.out[pix] = escaped ? (int32_t)o.wz : 0;
                    if (rq.pl.mag)
                        rq.pl.mag[pix] = mp_mag<N>(o, mag);
                    done = true;
                } else {
#pragma unroll
                    for (int k = 0; k < N; ++k) {
                        sp[k] = o.wre[k];
                        sp[N + k] = o.wim[k];
                    }
                    sp[2 * N] = o.wz + 1u;
                    sp[2 * N + 1] = (o.sre & 1u) | (o.sim & 2u);
                    again = true;
                }
            }
        }
        // warp-aggregated append of the unfinished pixels
        const unsigned amask = __ballot_sync(0xffffffffu, again);
        if (amask) {
            const int leader = __ffs(amask) - 1;
            unsigned b = 0;
            if (lane == leader)
                b = atomicAdd(qout_count, (unsigned)__popc(amask));
            b = __shfl_sync(0xffffffffu, b, leader);
            if (again)
                qout[b + __popc(amask & ((1u << lane) - 1u))] = e & ~kEntryFresh;
        }
        const unsigned dmask = __ballot_sync(0xffffffffu, done);
        if (done) {
            const unsigned grp = __match_any_sync(dmask, slot);
            if (lane == __ffs(grp) - 1)
                atomicSub(d->status.remaining + slot, (unsigned)__popc(grp));
        }
    }
}

// Dynamic shared memory of a frame block: c, above 16 words.
template <int N>
constexpr size_t frame_smem()
{
    return c_in_smem<N>() ? (size_t)2 * N * frame_block<N>() * sizeof(uint32_t) : 0;
}

// Lets a frame kernel have its shared memory (with the static part it passes
// the 48 KB that need no leave from 20 words on).  The leave is the current
// device's, so every launch asks: a process may render on several.
template <int N, int FRACTAL, bool JULIA>
int allow_frame_smem()
{
    if (frame_smem<N>())
        MDZ_CUDA_TRY(cudaFuncSetAttribute(mp_frame_kernel<N, FRACTAL, JULIA>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)frame_smem<N>()));
    return MDZGPU_OK;
}

// Loads one frame kernel: with lazy module loading, a load waits for the work
// running on the device, so servers call it before they start.
template <int N, int FRACTAL, bool JULIA>
int load_frame_kernel()
{
    cudaFuncAttributes a;
    MDZ_CUDA_TRY(cudaFuncGetAttributes(&a, mp_frame_kernel<N, FRACTAL, JULIA>));
    return allow_frame_smem<N, FRACTAL, JULIA>();
}

template <int N>
int pixel_blocks_per_sm(int* out)
{
    static int blocks_per_sm = 0;
    if (!blocks_per_sm) {
        int b = 0;
        MDZ_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, mp_pixel_kernel<N>,
                                                                   pixel_threads<N>(), 0));
        blocks_per_sm = b < 1 ? 1 : b;
    }
    *out = blocks_per_sm;
    return MDZGPU_OK;
}

template <int N, int FRACTAL, bool JULIA>
int launch_typed(mdzgpu_ctx* ctx, const MpLaunch& p, cudaStream_t s)
{
    constexpr int threads = frame_block<N>();
    if (int rc = allow_frame_smem<N, FRACTAL, JULIA>())
        return rc;
    const long tiles = p.list ? ((long)p.W * p.nrows + 31) / 32
                              : (long)((p.W + kTileW - 1) / kTileW) * ((p.nrows + kTileH - 1) / kTileH);
    long grid = ctx->num_sms;   // a block an SM
    const long blocks_needed = std::max((tiles + threads / 32 - 1) / (threads / 32),
                                        std::min(tiles, (long)ctx->num_sms));
    if (grid > blocks_needed)
        grid = blocks_needed;
    if (grid < 1)
        grid = 1;
    mp_frame_kernel<N, FRACTAL, JULIA><<<(unsigned)grid, threads, frame_smem<N>(), s>>>(p);
    MDZ_CUDA_TRY(cudaGetLastError());
    return MDZGPU_OK;
}

}  // namespace

template <int N>
int launch_words(mdzgpu_ctx* ctx, const MpLaunch& frame, cudaStream_t s)
{
    MpLaunch p = frame;
    p.pixel_limit = p.split_limit = 0;
    // The kernels look at the list's length, which only the device knows, and
    // all but one of them leave; a short list is done in the first chunk (a
    // later chunk means it was longer than the first one).
    if constexpr (split_list_per_sm<N>() > 0) {
        if (p.list && p.tile_base == 0) {
            p.pixel_limit = (unsigned)(pixel_list_per_sm<N>() * ctx->num_sms);
            p.split_limit = (unsigned)(split_list_per_sm<N>() * ctx->num_sms);
            if constexpr (pixel_list_per_sm<N>() > 0) {
                constexpr int threads = pixel_threads<N>();
                int b = 0;
                if (int rc = pixel_blocks_per_sm<N>(&b))
                    return rc;
                const long pixels = std::min((long)p.W * p.nrows, (long)p.pixel_limit);
                mp_pixel_kernel<N>
                    <<<(unsigned)std::min(pixels, (long)ctx->num_sms * b), threads, 0, s>>>(p);
                MDZ_CUDA_TRY(cudaGetLastError());
            }
            // (32 pixels a block; the blocks do not wait for one another)
            mp_split_kernel<N><<<(unsigned)(split_list_per_sm<N>() / 32 * ctx->num_sms),
                                 kSplitBlock, 0, s>>>(p, (unsigned)ctx->num_sms);
            MDZ_CUDA_TRY(cudaGetLastError());
        }
    }
    const bool julia = p.family == MDZ_FAMILY_JULIA;
    switch (p.fractal) {
    case MDZ_BURNING_SHIP:
        return julia ? launch_typed<N, MDZ_BURNING_SHIP, true>(ctx, p, s)
                     : launch_typed<N, MDZ_BURNING_SHIP, false>(ctx, p, s);
    case MDZ_GENERALIZED_CELTIC:
        return julia ? launch_typed<N, MDZ_GENERALIZED_CELTIC, true>(ctx, p, s)
                     : launch_typed<N, MDZ_GENERALIZED_CELTIC, false>(ctx, p, s);
    case MDZ_VARIANT:
        return julia ? launch_typed<N, MDZ_VARIANT, true>(ctx, p, s)
                     : launch_typed<N, MDZ_VARIANT, false>(ctx, p, s);
    default:
        return julia ? launch_typed<N, MDZ_MANDELBROT, true>(ctx, p, s)
                     : launch_typed<N, MDZ_MANDELBROT, false>(ctx, p, s);
    }
}


template <int N>
int launch_serve_mp_words(ServeDev* d, int mp_class, int num_sms, cudaStream_t s)
{
    constexpr int threads = block_threads<N>();
    const size_t smem = c_in_smem<N>() ? (size_t)2 * N * threads * sizeof(uint32_t) : 0;
    static int bps = 0;
    if (!bps) {
        if (smem > 48 * 1024)
            MDZ_CUDA_TRY(cudaFuncSetAttribute(serve_mp_kernel<N>,
                                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)smem));
        MDZ_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, serve_mp_kernel<N>,
                                                                   threads, smem));
        if (bps < 1)
            bps = 1;
    }
    serve_mp_kernel<N><<<(unsigned)(num_sms * bps), threads, smem, s>>>(d, mp_class);
    MDZ_CUDA_TRY(cudaGetLastError());
    return MDZGPU_OK;
}

template <int N>
int preload_words()
{
    int b = 0, rc = MDZGPU_OK;
    if constexpr (pixel_list_per_sm<N>() > 0)
        rc = pixel_blocks_per_sm<N>(&b);
    if constexpr (split_list_per_sm<N>() > 0) {
        if (!rc)
            MDZ_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, mp_split_kernel<N>,
                                                                       kSplitBlock, 0));
    }
    for (int j = 0; j < 2 && !rc; ++j) {
        const bool julia = j == 1;
        rc = julia ? load_frame_kernel<N, MDZ_MANDELBROT, true>()
                   : load_frame_kernel<N, MDZ_MANDELBROT, false>();
        if (!rc)
            rc = julia ? load_frame_kernel<N, MDZ_BURNING_SHIP, true>()
                       : load_frame_kernel<N, MDZ_BURNING_SHIP, false>();
        if (!rc)
            rc = julia ? load_frame_kernel<N, MDZ_GENERALIZED_CELTIC, true>()
                       : load_frame_kernel<N, MDZ_GENERALIZED_CELTIC, false>();
        if (!rc)
            rc = julia ? load_frame_kernel<N, MDZ_VARIANT, true>()
                       : load_frame_kernel<N, MDZ_VARIANT, false>();
    }
    return rc;
}

#ifdef MDZ_MP_WORDS
// One translation unit per word count (the build compiles this file once for
// every count in the list) keeps the large unrolled kernels compiling in
// parallel.
template int launch_words<MDZ_MP_WORDS>(mdzgpu_ctx*, const MpLaunch&, cudaStream_t);
template int launch_serve_mp_words<MDZ_MP_WORDS>(ServeDev*, int, int, cudaStream_t);
template int preload_words<MDZ_MP_WORDS>();
#endif

}  // namespace mdz
