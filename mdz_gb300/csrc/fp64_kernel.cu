// FP64 escape-time kernel: the GPU form of MDZ's hardware-float path.
//
// Arithmetic follows, operation for operation, the reference built with
// `long double` = IEEE double and no FMA contraction:
//   pixel -> coordinate  src/fractal.c:50-77
//   Mandelbrot           src/frac_mandel.c:5-21
//   burning ship         src/frac_burning_ship.c:7-24
//   generalized celtic   src/frac_generalized_celtic.c:7-24
//   mandel-celtic hybrid src/frac_variant.c:5-24
// Every value is the IEEE double the reference's operation gives, so the
// counts are bit-exact whatever -fmad says.
//
// What bounds it: the FP64 pipe, one warp instruction per 16 (DFMA) to 19
// (DADD, DMUL) cycles of an SM, where an integer instruction takes about
// half a cycle.  So an iteration spends three FP64 instructions, all DFMA:
// the three additions (a + b = fma(a, 1, b); 2 wre wim + c_im in one, the
// doubling being exact), and forms its three products on the integer pipes,
// bit for bit as the FP64 pipe would (double_bits.cuh); the escape test compares
// 20-bit magnitudes and adds in double only near the bailout.  Measured
// (960x540, 5.4e9 pixel-iterations): 168.6 ms with the nine FP64
// instructions this replaces and whole tiles, 40.4 ms now; 122 warp
// instructions an iteration, 65 SM cycles, the FP64 pipe 74% busy.
//
// An orbit whose (wre, wim) returns, bit for bit, to an earlier value repeats
// for ever and never escapes: the pixel's count is 0 whatever the depth.  Each
// iteration compares the state with the one kept at the last power of two
// (Brent's cycle search); a pixel inside an attracting cycle's basin
// converges to its cycle in a few hundred iterations.
//
// Work split (the GPU form of src/render_threads.c:360-393): warps pull 8x4
// pixel tiles from a global atomic counter, in place of a mutex-protected
// next_line counter advanced by whole rows, and a lane takes a new pixel as
// soon as kRefill lanes are idle (pixel_feed.cuh).
#include <math.h>

#include <algorithm>

#include "double_bits.cuh"
#include "internal.h"
#include "pixel_feed.cuh"

namespace mdz {
namespace {

constexpr int kBlock = 128;
constexpr int kRefill = 3;        // idle lanes that make a warp take new pixels
constexpr int kRefillEvery = 4;   // iterations between looks at the idle lanes
// 16 warps an SM keep the FP64 pipe as busy as 32 do and take twice the tiles
// each, so fewer lanes idle at the frame's end (960x540 to depth 20000 around
// a boundary point: 40.4 ms with 16 warps, 42.4 with 24, 46.6 with 32, 46.7
// with 10; refill at 3 idle lanes 40.4 ms, at 6 42.0 ms).
constexpr int kBlocksPerSm = 4;

// A double's high word as a float cut to 20 bits: right for 2^-126 .. 2^128;
// of a smaller or larger one only the bits' sign and pattern are left.
__device__ __forceinline__ float cut20(double x)
{
    return __int_as_float((int)((uint32_t)__double2hiint(x) * 8u - 0xc0000000u));
}

// One pixel's orbit between iterations.
struct Orbit {
    double wre, wim, wre2, wim2;
    double c_re, c_im;
    double kre, kim;      // state kept for the cycle search
    Split r, i;           // of wre, wim
    uint32_t wz;          // iterations done
    uint32_t event;       // iteration after which the state is kept, or depth
    bool odd;             // a component's exponent is odd: next product in double
};

__device__ __forceinline__ void orbit_start(Orbit& o, double x, double y, double c_re, double c_im,
                                            uint32_t depth)
{
    o.wre = o.kre = x;
    o.wim = o.kim = y;
    o.c_re = c_re;
    o.c_im = c_im;
    o.wz = 0;
    o.event = min(2u, depth);
    o.r = split(x);
    o.i = split(y);
    o.odd = odd_exponent(o.r, o.i);
    o.wre2 = __dmul_rn(x, x);
    o.wim2 = __dmul_rn(y, y);
}

// The iteration as the reference writes it, in double throughout: z and its
// squares after iteration o.wz from (re, im, re2, im2).
template <int FRACTAL>
__device__ __forceinline__ void orbit_step_double(Orbit& o, double re, double im, double re2,
                                                  double im2)
{
    const double t = FRACTAL == MDZ_BURNING_SHIP ? __dmul_rn(2.0, fabs(__dmul_rn(re, im)))
                                                 : __dmul_rn(__dmul_rn(2.0, re), im);
    double d = __dsub_rn(re2, im2);
    if (FRACTAL == MDZ_GENERALIZED_CELTIC || (FRACTAL == MDZ_VARIANT && (o.wz & 1u)))
        d = fabs(d);
    o.wim = __dadd_rn(t, o.c_im);
    o.wre = __dadd_rn(d, o.c_re);
    o.r = split(o.wre);
    o.i = split(o.wim);
    o.odd = odd_exponent(o.r, o.i);
    o.wim2 = __dmul_rn(o.wim, o.wim);
    o.wre2 = __dmul_rn(o.wre, o.wre);
}

// The next iteration.  Returns true when the pixel is done, with its count.
template <int FRACTAL>
__device__ __forceinline__ bool orbit_step(Orbit& o, uint32_t depth, double one, double two,
                                           uint32_t& count)
{
    uint32_t hi, lo;
    const double re = o.wre, im = o.wim, re2 = o.wre2, im2 = o.wim2;
    ++o.wz;
    bool hard = mul_round(o.r, o.i, hi, lo) | o.odd;
    if (FRACTAL == MDZ_BURNING_SHIP)
        hi &= 0x7fffffffu;
    // 2.0 * wre * wim + c_im, burning ship 2.0 * fabsl(wre * wim) + c_im
    o.wim = dfma(__hiloint2double((int)hi, (int)lo), two, o.c_im);
    double d = dfma(im2, -one, re2);
    if (FRACTAL == MDZ_GENERALIZED_CELTIC || (FRACTAL == MDZ_VARIANT && (o.wz & 1u)))
        d = __hiloint2double(__double2hiint(d) & 0x7fffffff, __double2loint(d));
    o.wre = dfma(d, one, o.c_re);
    o.r = split(o.wre);
    o.i = split(o.wim);
    o.odd = odd_exponent(o.r, o.i);
    hard |= sqr_round(o.i, hi, lo) | o.odd;
    o.wim2 = __hiloint2double((int)hi, (int)lo);
    hard |= sqr_round(o.r, hi, lo);
    o.wre2 = __hiloint2double((int)hi, (int)lo);
    if (hard)   // one lane in ~10^6, and zeros
        orbit_step_double<FRACTAL>(o, re, im, re2, im2);
    // |z|^2 > 4: a cut is below its value by at most 2^-20 of it; of a value
    // below 2^-126 it is some positive number or NaN, which hides no escape
    if (!(fabsf(cut20(o.wim2)) + fabsf(cut20(o.wre2)) <= 3.9999f) || hard) {
        double m;   // volatile: computed here only
        asm volatile("add.rn.f64 %0, %1, %2;" : "=d"(m) : "d"(o.wim2), "d"(o.wre2));
        if (m > 4.0) {
            count = o.wz;
            return true;
        }
    }
    // the states kept are the start's and those after iterations 2, 4, 8, ..,
    // so the hybrid's formula agrees too when wz is even
    if (((__double2loint(o.wre) ^ __double2loint(o.kre))
         | (__double2loint(o.wim) ^ __double2loint(o.kim)))
        == 0) {
        if (__double2hiint(o.wre) == __double2hiint(o.kre)
            && __double2hiint(o.wim) == __double2hiint(o.kim)
            && (FRACTAL != MDZ_VARIANT || (o.wz & 1u) == 0u)) {
            count = 0;
            return true;
        }
    }
    if (o.wz == o.event) {
        if (o.wz >= depth) {
            count = 0;
            return true;
        }
        o.kre = o.wre;
        o.kim = o.wim;
        o.event = min(o.event * 2u, depth);
    }
    return false;
}

// A pixel on the real axis (z_0 and c real) stays there: wim is a zero, whose
// sign nothing depends on, and every formula is wre = wre^2 + c_re.  A view
// centred on the axis has a row of them.
__device__ __forceinline__ bool on_axis(double y, double c_im)
{
    return (((hi_of(y) | hi_of(c_im)) & 0x7fffffff) | __double2loint(y) | __double2loint(c_im)) == 0;
}

// orbit_step there: one FP64 instruction.  (orbit_step forms the products of a
// zero in double, ten FP64 instructions more: 240x180 of the whole set to depth
// 1000, a row on the axis, 0.67 ms, 0.48 so; 2000 pixel-iterations alone 1.19 ms
// and 0.35.)
__device__ __forceinline__ bool orbit_step_axis(Orbit& o, uint32_t depth, double one,
                                                uint32_t& count)
{
    ++o.wz;
    o.wre = dfma(o.wre2, one, o.c_re);
    o.wre2 = sqr_bits(o.wre);
    // wre^2 > 4, and not NaN
    if ((uint64_t)__double_as_longlong(o.wre2) - 0x4010000000000001ull
        <= 0x7ff0000000000000ull - 0x4010000000000001ull) {
        count = o.wz;
        return true;
    }
    if (__double_as_longlong(o.wre) == __double_as_longlong(o.kre)) {
        count = 0;
        return true;
    }
    if (o.wz == o.event) {
        if (o.wz >= depth) {
            count = 0;
            return true;
        }
        o.kre = o.wre;
        o.event = min(o.event * 2u, depth);
    }
    return false;
}

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// AXIS: a row of the frame is on the real axis.
template <int FRACTAL, bool JULIA, bool AXIS>
__global__ void __launch_bounds__(kBlock) fp64_frame_kernel(Fp64Launch p)
{
    // the warp's current tile
    struct Pixel {
        double x, y;
        int ix, row;
    };
    __shared__ Pixel tile[kBlock / 32][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tiles_x = (p.W + kTileW - 1) / kTileW;
    const int tiles_y = (p.nrows + kTileH - 1) / kTileH;
    const unsigned total = (unsigned)tiles_x * (unsigned)tiles_y;
    const double width = __dsub_rn(p.xmax, p.xmin);
    const double fw = (double)p.W;
    const double ystep = __ddiv_rn(width, fw);
    unsigned long long its = 0;
    TileFeed feed;
    bool active = false;           // this lane iterates a pixel
    int ix = 0, lrow = 0;          // (~lrow for a pixel of the real axis)
    int band = -1;
    Orbit o;
    for (;;) {
        if (p.tile_rows_done)
            count_bands(p.W, p.nrows, p.tile_rows_done, p.band_flags, band);
        feed_lanes(
            feed, !active,
            [&]() {
                const unsigned t = next_tile(feed, &p.sync->tile_counter, p.stop);
                return t < total ? t : ~0u;
            },
            [&](unsigned t, int& px, int& row) {
                const int ty = (int)(t / (unsigned)tiles_x);
                px = (int)(t - (unsigned)ty * (unsigned)tiles_x) * kTileW + (lane & (kTileW - 1));
                row = ty * kTileH + lane / kTileW;
                return px < p.W && row < p.nrows;
            },
            [&](int k, int px, int row) {
                const double y = __dsub_rn(p.ymax, __dmul_rn(ystep, (double)(p.row0 + row)));
                const double x = __dadd_rn(__dmul_rn(__ddiv_rn((double)px, fw), width), p.xmin);
                tile[warp][k] = Pixel{x, y, px, row};
            },
            [&](int k) {
                const Pixel& q = tile[warp][k];
                ix = q.ix;
                lrow = q.row;
                orbit_start(o, q.x, q.y, JULIA ? p.jre : q.x, JULIA ? p.jim : q.y, p.depth);
                if (AXIS && on_axis(q.y, o.c_im))
                    lrow = ~lrow;
                active = true;
            });
        if (!__any_sync(0xffffffffu, active))
            break;
        // iterate until enough lanes are idle to be worth a look
        const int enough = (feed.left || feed.more) ? kRefill : 32;
        do {
            if (active) {
                uint32_t n;
                int u = kRefillEvery;
                bool done;
                if (AXIS && lrow < 0) {
#pragma unroll 1
                    do
                        done = orbit_step_axis(o, p.depth, p.one, n);
                    while (!done && --u);
                } else {
#pragma unroll 1
                    do
                        done = orbit_step<FRACTAL>(o, p.depth, p.one, p.two, n);
                    while (!done && --u);
                }
                if (done) {
                    if (AXIS && lrow < 0)
                        lrow = ~lrow;
                    p.out[(size_t)lrow * p.W + ix] = (int32_t)n;
                    its += n ? n : p.depth;
                    active = false;
                    band = lrow / kTileH;
                }
            }
        } while (__popc(__ballot_sync(0xffffffffu, !active)) < enough);
    }
    its = warp_sum_u64(its);
    if (lane == 0 && its)
        atomicAdd(&p.sync->iter_sum, its);
}

template <int FRACTAL, bool JULIA, bool AXIS>
int launch_one(mdzgpu_ctx* ctx, const Fp64Launch& p, cudaStream_t s)
{
    static int blocks_per_sm = 0;
    if (!blocks_per_sm) {
        MDZ_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &blocks_per_sm, fp64_frame_kernel<FRACTAL, JULIA, AXIS>, kBlock, 0));
        if (blocks_per_sm < 1)
            blocks_per_sm = 1;
    }
    const long tiles = (long)((p.W + kTileW - 1) / kTileW) * ((p.nrows + kTileH - 1) / kTileH);
    long grid = (long)ctx->num_sms * (blocks_per_sm < kBlocksPerSm ? blocks_per_sm : kBlocksPerSm);
    // a warp a tile, or fewer; a block an SM as long as there are tiles
    const long blocks_needed = std::max((tiles + kBlock / 32 - 1) / (kBlock / 32),
                                        std::min(tiles, (long)ctx->num_sms));
    if (grid > blocks_needed)
        grid = blocks_needed;
    if (grid < 1)
        grid = 1;
    fp64_frame_kernel<FRACTAL, JULIA, AXIS><<<(unsigned)grid, kBlock, 0, s>>>(p);
    MDZ_CUDA_TRY(cudaGetLastError());
    return MDZGPU_OK;
}

// Whether a row of the frame is on the real axis.  (Both kernels give the same
// counts there; the test for such a pixel costs the other frames 0.4%: the
// 2877x1623 Julia picture 2.295 ms and 2.286.)
bool has_axis_row(const Fp64Launch& p)
{
    if (p.family == MDZ_FAMILY_JULIA && p.jim != 0.0)
        return false;
    const double step = (p.xmax - p.xmin) / (double)p.W;
    const double k = p.ymax == 0.0 ? 0.0 : nearbyint(p.ymax / step);
    if (!(k >= (double)p.row0 - 2.0 && k <= (double)p.row0 + (double)p.nrows + 1.0))
        return false;
    for (long line = (long)k - 2; line <= (long)k + 2; ++line) {
        volatile const double down = step * (double)line;   // rounded, as the kernel's
        if (line >= p.row0 && line < (long)p.row0 + p.nrows && p.ymax - down == 0.0)
            return true;
    }
    return false;
}

template <int FRACTAL>
int launch_formula(mdzgpu_ctx* ctx, const Fp64Launch& p, cudaStream_t s)
{
    const bool axis = has_axis_row(p);
    if (p.family == MDZ_FAMILY_JULIA)
        return axis ? launch_one<FRACTAL, true, true>(ctx, p, s)
                    : launch_one<FRACTAL, true, false>(ctx, p, s);
    return axis ? launch_one<FRACTAL, false, true>(ctx, p, s)
                : launch_one<FRACTAL, false, false>(ctx, p, s);
}

}  // namespace

int launch_fp64(mdzgpu_ctx* ctx, const Fp64Launch& p, cudaStream_t s)
{
    switch (p.fractal) {
    case MDZ_BURNING_SHIP:
        return launch_formula<MDZ_BURNING_SHIP>(ctx, p, s);
    case MDZ_GENERALIZED_CELTIC:
        return launch_formula<MDZ_GENERALIZED_CELTIC>(ctx, p, s);
    case MDZ_VARIANT:
        return launch_formula<MDZ_VARIANT>(ctx, p, s);
    default:  // MANDELBROT and anything else, as the reference's `default:`
        return launch_formula<MDZ_MANDELBROT>(ctx, p, s);
    }
}

}  // namespace mdz
