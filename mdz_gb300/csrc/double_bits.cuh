// IEEE double products on the integer pipes, and decisions about doubles
// from their bits: this GPU's FP64 pipe takes 16 (DFMA) to 19 (DADD, DMUL,
// DSETP) cycles of an SM for a warp instruction, the integer pipes about
// half a cycle (1.1 for a 32x32->64 multiply-add).  A product rounded here
// takes about 14 instructions and gives the FP64 pipe's result bit for bit.
#pragma once

#include <stdint.h>

namespace mdz {

// a b + c, never simplified to an addition or a product
__device__ __forceinline__ double dfma(double a, double b, double c)
{
    double r;
    asm("fma.rn.f64 %0, %1, %2, %3;" : "=d"(r) : "d"(a), "d"(b), "d"(c));
    return r;
}

// A double cut in three: its mantissa with the leading 1 (h: top 21 bits,
// l: low 32) and q = high word - h, its sign and exponent field less one.
struct Split {
    uint32_t h, l, q;
};

__device__ __forceinline__ Split split(double x)
{
    const uint32_t hi = (uint32_t)__double2hiint(x);
    const uint32_t h = (hi & 0x000fffffu) | 0x00100000u;
    return Split{h, (uint32_t)__double2loint(x), hi - h};
}

// Whether one of the two has an exponent outside 2^-479 .. 2^32 (0,
// denormals, infinities and NaN are outside): inside, no product of the two
// leaves the normal range, and its magnitude fits a float's exponent.  The
// sign bit falls out of the mask.
__device__ __forceinline__ bool odd_exponent(const Split& x, const Split& y)
{
    const uint32_t lowest = 0x22000000u - 0x00100000u;
    return (((x.q - lowest) | (y.q - lowest)) & 0x60000000u) != 0u;
}

// x y rounded to nearest from the product of the mantissas, H 2^64 + m 2^32 +
// t (t's low word is not needed); q is the sum of the operands' q.  Returns
// true when the bits below the result's last place are 100..0 as far as m
// goes: t or the parity decides there, and the caller multiplies in double.
__device__ __forceinline__ bool round106(uint64_t H, uint64_t m, uint64_t t, uint32_t q,
                                         uint32_t& hi, uint32_t& lo)
{
    uint32_t v, hl, hh;   // bits 32.., 64.., 96.. of the product
    asm("{add.cc.u32 %0, %3, %4;\n\t"
        "addc.cc.u32 %1, %5, %6;\n\t"
        "addc.u32 %2, %7, 0;}"
        : "=&r"(v), "=&r"(hl), "=r"(hh)
        : "r"((uint32_t)m), "r"((uint32_t)(t >> 32)), "r"((uint32_t)H), "r"((uint32_t)(m >> 32)),
          "r"((uint32_t)(H >> 32)));
    const uint32_t s = hh >> 9;          // 1: the mantissas' product is 2 or more
    const uint32_t sh = 12u - s;
    const uint32_t r = v << sh;          // what is rounded away
    asm("{.reg .u32 c;\n\t"
        "add.cc.u32 c, %2, %2;\n\t"      // carry = r >> 31: round up
        "addc.cc.u32 %0, %3, 0;\n\t"
        "addc.u32 %1, %4, %5;}"
        : "=&r"(lo), "=r"(hi)
        : "r"(r), "r"(__funnelshift_l(v, hl, sh)), "r"(__funnelshift_l(hl, hh, sh)),
          "r"(q + (s << 20) + (0x00200000u - 0x40000000u)));
    return r == 0x80000000u;
}

__device__ __forceinline__ uint64_t wide(uint32_t a, uint32_t b)
{
    return (uint64_t)a * b;
}

__device__ __forceinline__ bool mul_round(const Split& x, const Split& y, uint32_t& hi,
                                          uint32_t& lo)
{
    return round106(wide(x.h, y.h), wide(x.h, y.l) + wide(y.h, x.l), wide(x.l, y.l), x.q + y.q, hi,
                    lo);
}

__device__ __forceinline__ bool sqr_round(const Split& x, uint32_t& hi, uint32_t& lo)
{
    return round106(wide(x.h, x.h), wide(2u * x.h, x.l), wide(x.l, x.l), 2u * x.q, hi, lo);
}

// High word of a double: orders non-negative doubles as their values.
__device__ __forceinline__ int hi_of(double x)
{
    return __double2hiint(x);
}

// Operations of a rare branch.  They are volatile, so that they are not
// computed ahead of it, and the branch is a loop that runs once (once()):
// a short block without one becomes predicated instructions, which take the
// FP64 pipe's time on every iteration with no lane active (measured in the
// perturbation's FP64 pass: 19 FP64 warp instructions an iteration, 7 of them
// such).
__device__ __forceinline__ double mul_here(double x, double y)
{
    double r;
    asm volatile("mul.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(x), "d"(y));
    return r;
}
__device__ __forceinline__ double add_here(double x, double y)
{
    double r;
    asm volatile("add.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(x), "d"(y));
    return r;
}
__device__ __forceinline__ double fma_here(double x, double y, double z)
{
    double r;
    asm volatile("fma.rn.f64 %0, %1, %2, %3;" : "=d"(r) : "d"(x), "d"(y), "d"(z));
    return r;
}
__device__ __forceinline__ bool once()
{
    unsigned sm;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
    return sm == 0xffffffffu;   // no SM has this number
}

// x 2^K (K small and positive), by the exponent.
template <int K>
__device__ __forceinline__ double times_pow2(double x)
{
    const int h = __double2hiint(x);
    double r = __hiloint2double(h + (K << 20), __double2loint(x));
    if ((h & 0x7ff00000) == 0)   // 0 and denormals
        do
            r = mul_here(x, (double)(1 << K));
        while (once());
    return r;
}

// ldexp(x, k), by the exponent where x and the result are normal.
__device__ __forceinline__ double ldexp_bits(double x, int k)
{
    const int h = __double2hiint(x);
    const int ex = (h >> 20) & 0x7ff;
    if (ex != 0 && ex != 0x7ff && ex + k > 0 && ex + k < 0x7ff)
        return __hiloint2double(h + k * (1 << 20), __double2loint(x));
    return x == 0.0 ? x : ldexp(x, k);
}

// ilogb(x) of x != 0.
__device__ __forceinline__ int ilogb_bits(double x)
{
    const int ex = (__double2hiint(x) >> 20) & 0x7ff;
    return (ex != 0 && ex != 0x7ff) ? ex - 1023 : ilogb(x);
}

// x (2 y) rounded to nearest.
__device__ __forceinline__ double mul2_bits(double x, double y)
{
    const Split a = split(x), b = split(y);
    uint32_t hi, lo;
    const bool tie = mul_round(a, b, hi, lo);
    double r = __hiloint2double((int)(hi + 0x00100000u), (int)lo);
    if (tie | odd_exponent(a, b))
        do
            r = mul_here(x, add_here(y, y));
        while (once());
    return r;
}

// x^2 rounded to nearest.
__device__ __forceinline__ double sqr_bits(double x)
{
    const Split a = split(x);
    uint32_t hi, lo;
    const bool tie = sqr_round(a, hi, lo);
    double r = __hiloint2double((int)hi, (int)lo);
    if (tie | odd_exponent(a, a))
        do
            r = mul_here(x, x);
        while (once());
    return r;
}

}  // namespace mdz
