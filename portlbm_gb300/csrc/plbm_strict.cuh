// plbm_strict.cuh — the F64_STRICT collision on the integer pipe.
//
// GB300 issues about two FP64 lanes per cycle and SM, 32 times fewer than 32-bit integer ones, and the
// reference's BGK update is 97 separately rounded FP64 operations a node: that alone took 48 cycles
// of an SM per node.  Most of those operations are sums of numbers of known, similar magnitude.
// Here they are done in 64-bit fixed point and rounded to 53 significant bits by hand, so every
// intermediate value is the IEEE double the reference computes: same operations, same order, each
// rounded once to nearest, ties to even.  What stays on the FP64 pipe (25 operations) are the
// products of two variables and the last relaxation step, whose operands have no common scale.
//
// Measured (k_nptl<F64_STRICT, STREAM>, 4096 x 4096): 5.7 k -> 17.7 k MLUPS; 2000 x 500: npol records
// 194 -> 72.4 us a step, nsol stream 194 -> 62.1 us.  With 25 FP64 instructions and about 780 on the ALU pipe
// a warp both pipes are 70 % busy (the plain sequence keeps the FP64 pipe full); each further
// operation moved off the FP64 pipe costs 12 to 30 ALU instructions against its 32 ALU slots' time.
// Converting |j| with I2F.F64 instead of by hand: 16.2 k; 4.5 a and 1.5 u^2 as FP64 products: 17.7 k.
//
// Fixed point: X = x * 2^61 in an int64.
//  * A double x in [2^-7, 2) is a multiple of 2^-59, so X is exact and a multiple of 4.
//  * Sums of such numbers are exact; rounding to 53 bits clears at most the low 10 bits (values below
//    4).  It is done by the FP32 adder (rne): the low 12 bits as a float, plus 2^(23+k), minus it
//    again, rounds them to a multiple of 2^k, ties to even, two instructions on a pipe that is
//    otherwise idle.
//  * An addend with bits below 2^-61 (a product from the FP64 pipe) enters with its lost bits ORed
//    into bit 0 (sticky): the other addend is a multiple of 4, so the sum lies on the same side of
//    every rounding boundary as the exact one as long as k >= 2, i.e. for sums of at least 2^-7.
//
// The fast path needs every population in [2^-7, 2), density and momentum in the range checked in
// `fast_collide` and |f - feq| < 2^-7; it says whether they were, and the caller otherwise runs the
// plain FP64 sequence on top.  That costs more than the sequence alone (2000 x 500, every node outside:
// 245 us a step against 197; a run that has diverged is such a case), so channels whose boundaries lead out of
// the range do without the fast path (strict_pays).  The code is shared with the host so that it can be compared with plain
// double arithmetic there.
#pragma once

#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define PLBM_HD __host__ __device__ __forceinline__
#else
#include <cmath>
#define PLBM_HD inline
#endif

namespace plbm {
namespace strict {

typedef unsigned long long u64;
typedef long long i64;

PLBM_HD uint32_t hi32(u64 x) { return (uint32_t)(x >> 32); }
PLBM_HD uint32_t lo32(u64 x) { return (uint32_t)x; }
PLBM_HD u64 join(uint32_t hi, uint32_t lo) { return ((u64)hi << 32) | lo; }

PLBM_HD u64 bits_of(double d)
{
#if defined(__CUDA_ARCH__)
    return (u64)__double_as_longlong(d);
#else
    u64 u; memcpy(&u, &d, 8); return u;
#endif
}
PLBM_HD double from_bits(u64 u)
{
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((i64)u);
#else
    double d; memcpy(&d, &u, 8); return d;
#endif
}
PLBM_HD float float_bits(uint32_t u)
{
#if defined(__CUDA_ARCH__)
    return __uint_as_float(u);
#else
    float f; memcpy(&f, &u, 4); return f;
#endif
}
PLBM_HD uint32_t bits_float(float f)
{
#if defined(__CUDA_ARCH__)
    return __float_as_uint(f);
#else
    uint32_t u; memcpy(&u, &f, 4); return u;
#endif
}
PLBM_HD float add_rn(float a, float b)
{
#if defined(__CUDA_ARCH__)
    return __fadd_rn(a, b);
#else
    volatile float r = a + b; return r;
#endif
}
PLBM_HD double mul_rn(double a, double b)
{
#if defined(__CUDA_ARCH__)
    return __dmul_rn(a, b);
#else
    volatile double r = a * b; return r;
#endif
}
PLBM_HD double plus_rn(double a, double b)
{
#if defined(__CUDA_ARCH__)
    return __dadd_rn(a, b);
#else
    volatile double r = a + b; return r;
#endif
}
PLBM_HD double fma_rn(double a, double b, double c)
{
#if defined(__CUDA_ARCH__)
    return __fma_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}
PLBM_HD int clz32(uint32_t x)
{
#if defined(__CUDA_ARCH__)
    return __clz((int)x);
#else
    return x ? __builtin_clz(x) : 32;
#endif
}
PLBM_HD uint32_t min_u(uint32_t a, uint32_t b) { return a < b ? a : b; }

// X rounded to a multiple of 2^k, nearest, ties to even, 1 <= k <= 11; kbits = (150 + k) << 23, the
// float 2^(23+k).  (float)2^23 + low is exact, adding 2^(23+k) leaves an ulp of 2^k, and every bit
// above the low 12 is an even multiple of 2^k.
PLBM_HD u64 round_low(u64 x, uint32_t kbits)
{
    const uint32_t v = (lo32(x) & 0xFFFu) | 0x4B000000u;
    const float big = float_bits(kbits);
    const uint32_t r = bits_float(add_rn(add_rn(float_bits(v), big), -big));
    return x + r - v;
}
// X >= 2^54 (and < 2^63) rounded to 53 significant bits: top bit p = 63 - clz, k = p - 52.
PLBM_HD u64 rne(u64 x)
{
    return round_low(x, (uint32_t)(161 - clz32(hi32(x))) << 23);
}
// Signed X, an even number: below 2^54 in magnitude it is already a 53-bit number and k = 1 leaves it.
// (For a negative X one's complement gives the magnitude's top bit, or one less at an exact power of
// two, which no rounding changes.)
PLBM_HD i64 rne_signed(i64 x)
{
    const uint32_t h = hi32((u64)x), m = h ^ (uint32_t)((int32_t)h >> 31);
    int e = 161 - clz32(m);
    if (e < 151) e = 151;
    return (i64)round_low((u64)x, (uint32_t)e << 23);
}

// A population: exact for a double in [2^-7, 2); `bad` collects what is outside that range.
PLBM_HD u64 to_fixed(double f, uint32_t &bad)
{
    const u64 b = bits_of(f);
    const uint32_t t = hi32(b) - (1016u << 20);      // exponent field 1016 .. 1023, sign 0
    bad |= t;                                        // any bit from 23 up: outside
    const int sh = (int)((t >> 20) & 7u) + 2;
    return join((hi32(b) & 0xFFFFFu) | 0x100000u, lo32(b)) << sh;
}

// RN(x * odd / 2) for a double x > 0 and odd = 3 or 9 on its mantissa: odd * M has two to four bits too
// many, rounded off with rne; the product's value is that times 2^(E - 1076).  (x = 0 gives some
// number below 2^-1021, as good as 0 to the callers.)
PLBM_HD double times_half(double x, uint32_t odd)
{
    const u64 b = bits_of(x);
    const u64 X = join((hi32(b) & 0xFFFFFu) | 0x100000u, lo32(b)) * odd;
    const int k = 11 - clz32(hi32(X));
    const u64 m = round_low(X, (uint32_t)(150 + k) << 23) >> k;
    return from_bits(m + join((hi32(b) & 0x7FF00000u) + ((uint32_t)(k - 2) << 20), 0));
}

// floor(x * 2^61) with the lost bits ORed into bit 0, for a double scaled by 2^122, 0 <= x < 1/2.
// x = 0 and x below 2^-61 give 1 (a positive number too small to matter).
PLBM_HD u64 to_sticky(double x122)
{
    const u64 b = bits_of(x122);
    const u64 m = join((hi32(b) << 11) | (lo32(b) >> 21) | 0x80000000u, lo32(b) << 11);
    const uint32_t n = min_u(1147u - (hi32(b) >> 20), 63u);      // unsigned: a NaN or a huge x clamps too
    const u64 x = m >> n;
    const u64 back = x << n;
    const uint32_t lost = (lo32(back) ^ lo32(m)) | (hi32(back) ^ hi32(m));
    return x | min_u(lost, 1u);
}

// RN(w * U) for U * 2^-61 the value and wq = w * 2^64 (a double w < 1 is a multiple of 2^-64 from 2^-11
// up): the 128-bit product's upper word on the same grid, its lower word as the sticky bit.
PLBM_HD u64 weigh(u64 U, uint32_t wh, uint32_t wl)
{
    const uint32_t uh = hi32(U), ul = lo32(U);
    const u64 p0 = (u64)ul * wl;
    const u64 p1 = (u64)ul * wh + hi32(p0);
    const u64 p2 = (u64)uh * wl + lo32(p1);
    const u64 p3 = (u64)uh * wh + hi32(p1) + hi32(p2);
    return rne(p3 | min_u(lo32(p0) | lo32(p2), 1u));
}

PLBM_HD int clz64(u64 x)
{
#if defined(__CUDA_ARCH__)
    return __clzll((i64)x);
#else
    return x ? __builtin_clzll(x) : 64;
#endif
}

// The magnitude of a multiple of 2^-61 of at most 53 significant bits, as the double |x| * 2^61.
PLBM_HD double magnitude(i64 x)
{
    const u64 s = (u64)(x >> 63), mag = ((u64)x ^ s) - s;
    const int z = clz64(mag);
    const u64 n = mag << (z & 63);
    return from_bits(mag ? (n >> 11) + join((uint32_t)(1085 - z) << 20, 0) : 0);
}

struct Fixed { i64 rho, jx, jy; double usq122; };   // moments: x * 2^61, and u^2 * 2^122

// The BGK update of collide_f64_strict for omega in [2^-500, 2^500].
// True when every value was in range; f then holds the new populations (f_out) and `m` the moments.
PLBM_HD bool fast_collide(const double f[9], double f_out[9], double omega, Fixed &m)
{
    uint32_t bad = 0;
    u64 F[9];
    for (int d = 0; d < 9; ++d) F[d] = to_fixed(f[d], bad);
    bad &= 0xFF800000u;
    u64 rho = F[0];
    for (int d = 1; d < 9; ++d) rho = rne(rho + F[d]);
    i64 jx = rne_signed((i64)(F[2] - F[0]));
    jx = rne_signed(jx - (i64)F[3]); jx = rne_signed(jx + (i64)F[5]);
    jx = rne_signed(jx - (i64)F[6]); jx = rne_signed(jx + (i64)F[8]);
    i64 jy = rne_signed(-(i64)F[0] - (i64)F[1]);
    jy = rne_signed(jy - (i64)F[2]); jy = rne_signed(jy + (i64)F[6]);
    jy = rne_signed(jy + (i64)F[7]); jy = rne_signed(jy + (i64)F[8]);
    {
        // with M = |jx| + |jy| < 0.2 and rho - 4 M >= 0.3, rho + 4 M < 2: every bracket
        // rho +- 3 cu, + 4.5 cu^2, - 1.5 u^2 lies in [0.3, 2) and every equilibrium in [2^-7, 1)
        const int32_t ax = (int32_t)hi32((u64)jx), ay = (int32_t)hi32((u64)jy), r = (int32_t)hi32(rho);
        const int32_t M = (ax ^ (ax >> 31)) + (ay ^ (ay >> 31)) + 2;
        const uint32_t one = 1u << 29;
        if ((uint32_t)M >= one / 5 || r < (int32_t)(one / 10 * 3) + 4 * M || (uint32_t)(r + 4 * M) >= 2 * one) bad = 1;
    }
    const double A = magnitude(jx), B = magnitude(jy);
    const double usq = plus_rn(mul_rn(A, A), mul_rn(B, B));
    const u64 h = to_sticky(times_half(usq, 3));
    const uint32_t w36h = 0x071C71C7u, w36l = 0x1C71C700u, w9h = 0x1C71C71Cu, w9l = 0x71C71C00u, w49h = 0x71C71C71u,
                   w49l = 0xC71C7000u;
    const i64 a[4] = { jx, jy, rne_signed(jx + jy), rne_signed(jx - jy) };
    // directions of +a and -a: jx 5/3, jy 7/1, jx+jy 8/0, jx-jy 2/6
    u64 feq[9];
    feq[4] = weigh(rne(rho - h), w49h, w49l);
#if defined(__CUDACC__)
#pragma unroll
#endif
    for (int k = 0; k < 4; ++k) {
        const double ad = k == 0 ? A : k == 1 ? B : magnitude(a[k]);
        const u64 c45 = to_sticky(mul_rn(times_half(ad, 9), ad));
        const i64 c3 = rne_signed(3 * a[k]);
        const u64 up = rne(rne(rne(rho + (u64)c3) + c45) - h), dn = rne(rne(rne(rho - (u64)c3) + c45) - h);
        const int dp = k == 0 ? 5 : k == 1 ? 7 : k == 2 ? 8 : 2;
        feq[dp] = weigh(up, k < 2 ? w9h : w36h, k < 2 ? w9l : w36l);
        feq[8 - dp] = weigh(dn, k < 2 ? w9h : w36h, k < 2 ? w9l : w36l);
    }
    // -omega (f - feq): the difference is exact, a multiple of 2^-59 (both are at least 2^-7), and below
    // 2^-7 its magnitude is the mantissa of 2^52 + |D|; the fused multiply-add of that rounds omega * |D|
    // once.  (An inlet 0.2 denser than the channel keeps its column just below that: with 2^-8 the column's
    // warps took both paths and a step of the 400 x 100 channel 8.2 us instead of 6.4.)
    const u64 ob = bits_of(omega);
    const double om = from_bits(ob - (59ull << 52)), omc = from_bits((ob - (7ull << 52)) ^ (1ull << 63));
    uint32_t far = 0;
#if defined(__CUDACC__)
#pragma unroll
#endif
    for (int d = 0; d < 9; ++d) {
        const i64 D = (i64)(F[d] - feq[d]) >> 2;                     // units of 2^-59
        const uint32_t s = (uint32_t)((int32_t)hi32((u64)D) >> 31);
        const u64 mag = ((u64)D ^ join(s, s)) - join(s, s);
        far |= hi32(mag);
        const double P = fma_rn(om, from_bits(mag | 0x4330000000000000ull), omc);
        const u64 pb = bits_of(P);
        f_out[d] = plus_rn(from_bits(join(hi32(pb) ^ (~s & 0x80000000u), lo32(pb))), f[d]);
    }
    bad |= far >> 20;
    m.rho = (i64)rho; m.jx = jx; m.jy = jy; m.usq122 = usq;
    return bad == 0;
}

}  // namespace strict
}  // namespace plbm
