// Multi-word fixed-point arithmetic for the deep-zoom kernels.
//
// A number is N 32-bit words (N even: N/2 64-bit limbs), two's complement,
// least significant word first, with F = 32*N - 8 fractional bits: 1 sign
// bit, 7 integer bits.  The iteration only ever holds |values| < 8 before a
// square (larger ones have already escaped) so squares stay below 64 and
// |z|^2 below 128: the format never overflows.
//
// Products are computed on magnitudes with PTX carry chains and truncated:
// partial products that land entirely below column N-2 are skipped.  Their
// sum is below N^2 * 2^(32(N-2)+64), i.e. below N^2 * 2^-24 units of the
// result's last place, so the truncated product is within 2 ulp of
// floor(a*b / 2^F).
//
// What bounds them is the integer multiplier: a 32x32->64 multiply-add takes
// a warp 1.1 cycles of an SM, and nothing else on this GPU multiplies integers
// faster.  A row a_i b of partial products is added as two chains, one of the
// products that start in even columns and one of those in odd columns, each
// into an accumulator of its own: within a chain the (low, high) halves of
// consecutive products are the words of one long number, so mad.lo.cc /
// madc.hi.cc pairs become one 64-bit multiply-add each, with the carry in
// and out of it (one chain of all low halves and one of all high halves, as
// here before, took two multiplications and two additions a product: N = 10
// general product 132 -> 87 cycles, N = 16 298 -> 174, N = 34 at one warp a
// scheduler 2035 -> 1028).  The two accumulators are added at the end.
#pragma once

#include <stdint.h>

namespace mdz {
namespace fx {

// One chain: x[0] b, x[2] b, ... added into e[0..1], e[2..3], ...; CNT
// products, CARRY: the carry out of the last goes to e[2 CNT], untouched so far.
template <int CNT, bool CARRY>
__device__ __forceinline__ void chain(uint32_t* e, const uint32_t* x, uint32_t b)
{
#pragma unroll
    for (int t = 0; t < CNT; ++t) {
        if (t == 0)
            asm volatile("mad.lo.cc.u32 %0, %1, %2, %0;" : "+r"(e[0]) : "r"(x[0]), "r"(b));
        else
            asm volatile("madc.lo.cc.u32 %0, %1, %2, %0;" : "+r"(e[2 * t]) : "r"(x[2 * t]), "r"(b));
        if (CARRY || t < CNT - 1)
            asm volatile("madc.hi.cc.u32 %0, %1, %2, %0;" : "+r"(e[2 * t + 1]) : "r"(x[2 * t]), "r"(b));
        else
            asm volatile("madc.hi.u32 %0, %1, %2, %0;" : "+r"(e[2 * t + 1]) : "r"(x[2 * t]), "r"(b));
    }
    if (CARRY)
        asm volatile("addc.u32 %0, 0, 0;" : "=r"(e[2 * CNT]));
}

// Column sums of a product, column N-2+k at index k: products that start in
// an even column in `even`, the others in `odd`.
template <int N>
struct Columns {
    uint32_t even[N + 4], odd[N + 4];
};

// Row I: a_j b for j = J0 .. N-1, into columns I + J0 .. I + N.  A chain
// that ends with j = N-1 carries nothing out (the sum of rows 0..I is below
// 2^(32 (I + 1 + N))); one that ends with j = N-2 carries into column I + N,
// where its accumulator is still zero.  (Both hold for any subset of the rows,
// taken in order.)
template <int N, int I, int J0>
__device__ __forceinline__ void row(Columns<N>& s, const uint32_t (&a)[N], uint32_t b)
{
    constexpr int k = I + J0 - (N - 2);
    constexpr int n0 = (N - 1 - J0) / 2 + 1, n1 = (N - 1 - J0 + 1) / 2;
    constexpr bool c0 = ((N - 1 - J0) & 1) != 0;   // the first chain ends with N-2
    if constexpr (k & 1) {
        chain<n0, c0>(s.odd + k, a + J0, b);
        if constexpr (n1 > 0)
            chain<n1, !c0>(s.even + k + 1, a + J0 + 1, b);
    } else {
        chain<n0, c0>(s.even + k, a + J0, b);
        if constexpr (n1 > 0)
            chain<n1, !c0>(s.odd + k + 1, a + J0 + 1, b);
    }
}

// rows I, I + STEP, ...
template <int N, int I, int STEP = 1>
__device__ __forceinline__ void mul_rows(Columns<N>& s, const uint32_t (&a)[N],
                                         const uint32_t (&b)[N])
{
    if constexpr (I < N) {
        row<N, I, (N - 2 - I > 0 ? N - 2 - I : 0)>(s, a, b[I]);
        mul_rows<N, I + STEP, STEP>(s, a, b);
    }
}

// off-diagonal products a_i a_j, i < j
template <int N, int I>
__device__ __forceinline__ void sqr_rows(Columns<N>& s, const uint32_t (&a)[N])
{
    if constexpr (I < N - 1) {
        constexpr int j0 = I + 1 > N - 2 - I ? I + 1 : N - 2 - I;
        if constexpr (j0 < N)
            row<N, I, j0>(s, a, a[I]);
        sqr_rows<N, I + 1>(s, a);
    }
}

// acc[k] = product column (N-2+k), k = 0..N+1, the two accumulators added.
template <int N>
__device__ __forceinline__ void add_columns(const Columns<N>& s, uint32_t (&acc)[N + 2])
{
    acc[0] = s.even[0];
    asm volatile("add.cc.u32 %0, %1, %2;" : "=r"(acc[1]) : "r"(s.even[1]), "r"(s.odd[1]));
#pragma unroll
    for (int k = 2; k < N + 1; ++k)
        asm volatile("addc.cc.u32 %0, %1, %2;" : "=r"(acc[k]) : "r"(s.even[k]), "r"(s.odd[k]));
    asm volatile("addc.u32 %0, %1, %2;" : "=r"(acc[N + 1]) : "r"(s.even[N + 1]), "r"(s.odd[N + 1]));
}

template <int N>
__device__ __forceinline__ void clear(Columns<N>& s)
{
#pragma unroll
    for (int k = 0; k < N + 4; ++k)
        s.even[k] = s.odd[k] = 0u;
}

// Truncated product of two magnitudes.
template <int N>
__device__ __forceinline__ void mul_trunc(const uint32_t (&a)[N], const uint32_t (&b)[N],
                                          uint32_t (&acc)[N + 2])
{
    Columns<N> s;
    clear(s);
    mul_rows<N, 0>(s, a, b);
    add_columns<N>(s, acc);
}

// The part of mul_trunc's sum from the rows of one parity; the two parts add
// up to it (add_part).
template <int N, int PARITY>
__device__ __forceinline__ void mul_part(const uint32_t (&a)[N], const uint32_t (&b)[N],
                                         uint32_t (&acc)[N + 2])
{
    Columns<N> s;
    clear(s);
    mul_rows<N, PARITY, 2>(s, a, b);
    add_columns<N>(s, acc);
}

// acc += the words part(0) .. part(N + 1)
template <int N, class Part>
__device__ __forceinline__ void add_part(uint32_t (&acc)[N + 2], const Part& part)
{
    asm volatile("add.cc.u32 %0, %0, %1;" : "+r"(acc[0]) : "r"(part(0)));
#pragma unroll
    for (int k = 1; k < N + 1; ++k)
        asm volatile("addc.cc.u32 %0, %0, %1;" : "+r"(acc[k]) : "r"(part(k)));
    asm volatile("addc.u32 %0, %0, %1;" : "+r"(acc[N + 1]) : "r"(part(N + 1)));
}

// Truncated square of a magnitude; acc as in mul_trunc.
template <int N>
__device__ __forceinline__ void sqr_trunc(const uint32_t (&a)[N], uint32_t (&acc)[N + 2])
{
    static_assert((N & 1) == 0, "diagonal products start in even columns");
    Columns<N> s;
    clear(s);
    sqr_rows<N, 0>(s, a);
    add_columns<N>(s, acc);
    // double
#pragma unroll
    for (int k = N + 1; k > 0; --k)
        acc[k] = __funnelshift_l(acc[k - 1], acc[k], 1);
    acc[0] <<= 1;
    // the diagonal: a_i^2 from column 2i on, 2i >= N-2 (column N-2 begins with
    // i = N/2 - 1), one chain
#pragma unroll
    for (int i = N / 2 - 1; i < N; ++i) {
        const int k = 2 * i - (N - 2);
        if (k == 0)
            asm volatile("mad.lo.cc.u32 %0, %1, %1, %0;" : "+r"(acc[k]) : "r"(a[i]));
        else
            asm volatile("madc.lo.cc.u32 %0, %1, %1, %0;" : "+r"(acc[k]) : "r"(a[i]));
        if (i < N - 1)
            asm volatile("madc.hi.cc.u32 %0, %1, %1, %0;" : "+r"(acc[k + 1]) : "r"(a[i]));
        else
            asm volatile("madc.hi.u32 %0, %1, %1, %0;" : "+r"(acc[k + 1]) : "r"(a[i]));
    }
}

// r = acc >> (F - s) restricted to N words: SH = 24 gives floor(P / 2^F),
// SH = 23 gives floor(2P / 2^F).
template <int N, int SH>
__device__ __forceinline__ void extract(const uint32_t (&acc)[N + 2], uint32_t (&r)[N])
{
#pragma unroll
    for (int k = 0; k < N; ++k)
        r[k] = __funnelshift_r(acc[1 + k], acc[2 + k], SH);
}

// r = c + (x ^ m) + (m & 1): c + x when m == 0, c - x when m == ~0.
template <int N, class CGet>
__device__ __forceinline__ void add_signed(const CGet& c, const uint32_t (&x)[N], uint32_t m,
                                           uint32_t (&r)[N])
{
    uint32_t dummy;
    asm volatile("add.cc.u32 %0, %1, 0xffffffff;" : "=r"(dummy) : "r"(m & 1u));
#pragma unroll
    for (int k = 0; k < N; ++k) {
        if (k < N - 1)
            asm volatile("addc.cc.u32 %0, %1, %2;" : "=r"(r[k]) : "r"(c(k)), "r"(x[k] ^ m));
        else
            asm volatile("addc.u32 %0, %1, %2;" : "=r"(r[k]) : "r"(c(k)), "r"(x[k] ^ m));
    }
    (void)dummy;
}

// r = a - b
template <int N>
__device__ __forceinline__ void sub(const uint32_t (&a)[N], const uint32_t (&b)[N], uint32_t (&r)[N])
{
    asm volatile("sub.cc.u32 %0, %1, %2;" : "=r"(r[0]) : "r"(a[0]), "r"(b[0]));
#pragma unroll
    for (int k = 1; k < N; ++k) {
        if (k < N - 1)
            asm volatile("subc.cc.u32 %0, %1, %2;" : "=r"(r[k]) : "r"(a[k]), "r"(b[k]));
        else
            asm volatile("subc.u32 %0, %1, %2;" : "=r"(r[k]) : "r"(a[k]), "r"(b[k]));
    }
}

// In place |x|; returns the sign mask (0 or ~0) of the input.
template <int N>
__device__ __forceinline__ uint32_t abs_inplace(uint32_t (&x)[N])
{
    const uint32_t m = (uint32_t)((int32_t)x[N - 1] >> 31);
    if constexpr (N <= 8) {
        // negation under a mask, 2 N additions: short enough that the branch
        // below costs more (3000 iterations of one pixel at 6 words 1.09 ms and
        // 1.17, a 320x240 frame 0.91 and 0.94; at 10 words a 256-bit frame
        // 19.4 ms and 18.9)
        uint32_t carry;
        asm volatile("add.cc.u32 %0, %1, 0xffffffff;" : "=r"(carry) : "r"(m & 1u));
#pragma unroll
        for (int k = 0; k < N; ++k) {
            if (k < N - 1)
                asm volatile("addc.cc.u32 %0, %1, 0;" : "=r"(x[k]) : "r"(x[k] ^ m));
            else
                asm volatile("addc.u32 %0, %1, 0;" : "=r"(x[k]) : "r"(x[k] ^ m));
        }
        (void)carry;
    } else if (m) {
        // a branch: N additions
        asm volatile("sub.cc.u32 %0, 0, %0;" : "+r"(x[0]));
#pragma unroll
        for (int k = 1; k < N; ++k) {
            if (k < N - 1)
                asm volatile("subc.cc.u32 %0, 0, %0;" : "+r"(x[k]));
            else
                asm volatile("subc.u32 %0, 0, %0;" : "+r"(x[k]));
        }
    }
    return m;
}

// |x| >= 8 (conservative on the negative side by less than 2^-24): the
// value has certainly escaped, and squaring it could overflow.
template <int N>
__device__ __forceinline__ bool big(const uint32_t (&x)[N])
{
    const int32_t top = (int32_t)x[N - 1];
    return top >= 0x08000000 || top < -0x08000000;
}

// a + b > 4 for non-negative a, b (< 64 each).
template <int N>
__device__ __forceinline__ bool sum_gt4(const uint32_t (&a)[N], const uint32_t (&b)[N])
{
    // the top words decide unless their sum is 4's or one below it
    const uint32_t t = a[N - 1] + b[N - 1];
    if (t - 0x03ffffffu > 1u)
        return t > 0x04000000u;
    uint32_t s[N];
    asm volatile("add.cc.u32 %0, %1, %2;" : "=r"(s[0]) : "r"(a[0]), "r"(b[0]));
#pragma unroll
    for (int k = 1; k < N; ++k) {
        if (k < N - 1)
            asm volatile("addc.cc.u32 %0, %1, %2;" : "=r"(s[k]) : "r"(a[k]), "r"(b[k]));
        else
            asm volatile("addc.u32 %0, %1, %2;" : "=r"(s[k]) : "r"(a[k]), "r"(b[k]));
    }
    uint32_t low = 0;
#pragma unroll
    for (int k = 0; k < N - 1; ++k)
        low |= s[k];
    const uint32_t top = s[N - 1];
    return top > 0x04000000u || (top == 0x04000000u && low != 0u);
}

}  // namespace fx
}  // namespace mdz
