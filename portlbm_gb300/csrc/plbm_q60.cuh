// plbm_q60.cuh — the products and the relaxation of the F64_Q60 collision (see plbm_device.cuh), shared with the
// host so that they can be compared with a plain formulation there.
#pragma once

#include "plbm_params.h"
#include "plbm_strict.cuh"   // PLBM_HD

namespace plbm {

PLBM_HD unsigned umulhi32(unsigned a, unsigned b)
{
#if defined(__CUDA_ARCH__)
    return __umulhi(a, b);
#else
    return (unsigned)((unsigned long long)a * b >> 32);
#endif
}
PLBM_HD int mulhi32(int a, int b)
{
#if defined(__CUDA_ARCH__)
    return __mulhi(a, b);
#else
    return (int)((long long)a * b >> 32);
#endif
}

// High 64 bits of the 128-bit product of unsigned a and b from three 32x32 partial products; the
// dropped low partial product and carries make it at most 2 units low.
PLBM_HD unsigned long long umulhi_approx(unsigned long long a, unsigned long long b)
{
    const unsigned al = (unsigned)a, ah = (unsigned)(a >> 32), bl = (unsigned)b, bh = (unsigned)(b >> 32);
    return (unsigned long long)ah * bh + umulhi32(ah, bl) + umulhi32(al, bh);
}

// c * v for a constant c in [0, 1) held as round(c * 2^64) and a Q60 value v; result Q60.
// POSITIVE: v >= 0, without the correction for a negative v.
template <bool POSITIVE = false>
PLBM_HD long long mulc(unsigned long long c, long long v)
{
    const unsigned long long r = umulhi_approx(c, (unsigned long long)v);
    return (long long)(!POSITIVE && v < 0 ? r - c : r);
}

// The same value for c <= 1/4 (omega / 8 and omega / 12 are; the rounded-up high half of c has to stay below 2^31)
// with v's high half signed: no correction is left (the 2^31 bit of c's low
// half moves into the high half's coefficient: floor(s (u + 2^32) / 2^32) = floor(s u / 2^32) + s).
PLBM_HD long long mulc_half(unsigned long long c, long long v)
{
    const unsigned ch = (unsigned)(c >> 32), cl = (unsigned)c;
    const int vh = (int)(v >> 32);
    return (long long)vh * (int)(ch + (cl >> 31)) + mulhi32(vh, (int)cl) + umulhi32((unsigned)v, ch);
}

// a * b for Q60 values with |a|, |b| < 2 (checked by the caller); result Q60.  The value of
// umulhi_approx corrected for negative operands, by signed high halves.
PLBM_HD long long mulv(long long a, long long b)
{
    const long long a2 = (long long)((unsigned long long)a << 2), b2 = (long long)((unsigned long long)b << 2);   // Q62
    const int ah = (int)(a2 >> 32), al = (int)a2, bh = (int)(b2 >> 32), bl = (int)b2;
    // floor(ah * (unsigned)bl / 2^32), and the same of bh and al
    const int m = mulhi32(ah, bl) + ((bl >> 31) & ah), n = mulhi32(bh, al) + ((al >> 31) & bh);
    return (long long)ah * bh + m + n;
}

// The BGK update of F64_FAST in Q60: f' = f - omega f + omega feq with
// omega feq_d = omega w_d (rho - 1.5 u^2) + 4.5 omega w_d cu^2 + 3 omega w_d cu.  Every constant is
// below 1 for relaxation_time > 0.5 and is applied with mulc; omega f uses omega/2 twice.  The ALU
// pipe bounds the kernels beside HBM: without the sign corrections that positive factors never need,
// and with the range tested on high words, a node takes 484 instead of 522 instructions (k_nptl,
// 4096 x 4096: ALU pipe 61 -> 45 % busy), the same values.  One step a launch, nptl stream: 8192 x 8192 1607 ->
// 1528 us, 2000 x 500 29.2 -> 26.3, 1024 x 256 8.6 -> 7.3 (with the dependent launches).  (Weights factored into powers
// of two times 1/9 need 12 constant products and reach 50.1 k, but round differently: |j| near rest,
// the square root of a few units of 2^-60, then moves by more than 1e-9.)
// POSITIVE: no population and no R below zero, nearly every node of a flow; 12 of the 20 constant
// products then need no correction for a negative factor.
template <bool POSITIVE>
PLBM_HD void relax_q60(long long f[9], long long jx, long long jy, long long jx2, long long jy2, long long jxy,
                       long long R, const StepParams &p)
{
    const unsigned long long wh = (unsigned long long)p.q_om1;   // omega / 2, Q64
    const long long usq = jx2 + jy2;
    const long long b9 = mulc<POSITIVE>((unsigned long long)p.q_ow9, R), b36 = mulc<POSITIVE>((unsigned long long)p.q_ow36, R);
    f[4] = f[4] + mulc<POSITIVE>((unsigned long long)p.q_ow49, R) - 2 * mulc<POSITIVE>(wh, f[4]);
    {
        const long long sym = mulc((unsigned long long)p.q_k9, jx2) + b9, ou = mulc((unsigned long long)p.q_o9, jx);
        f[5] = f[5] + sym + ou - 2 * mulc<POSITIVE>(wh, f[5]);
        f[3] = f[3] + sym - ou - 2 * mulc<POSITIVE>(wh, f[3]);
    }
    {
        const long long sym = mulc((unsigned long long)p.q_k9, jy2) + b9, ou = mulc((unsigned long long)p.q_o9, jy);
        f[7] = f[7] + sym + ou - 2 * mulc<POSITIVE>(wh, f[7]);
        f[1] = f[1] + sym - ou - 2 * mulc<POSITIVE>(wh, f[1]);
    }
    {
        const long long sym = mulc_half((unsigned long long)p.q_k36, usq + 2 * jxy) + b36;
        const long long ou = mulc_half((unsigned long long)p.q_o36, jx + jy);
        f[8] = f[8] + sym + ou - 2 * mulc<POSITIVE>(wh, f[8]);
        f[0] = f[0] + sym - ou - 2 * mulc<POSITIVE>(wh, f[0]);
    }
    {
        const long long sym = mulc_half((unsigned long long)p.q_k36, usq - 2 * jxy) + b36;
        const long long ou = mulc_half((unsigned long long)p.q_o36, jx - jy);
        f[2] = f[2] + sym + ou - 2 * mulc<POSITIVE>(wh, f[2]);
        f[6] = f[6] + sym - ou - 2 * mulc<POSITIVE>(wh, f[6]);
    }
}

// Whether a population left [-4, 4) or a momentum [-2, 2), by their high words: an offset makes the top bits of a
// value in range zero.
PLBM_HD bool q60_out_of_range(const long long f[9], long long jx, long long jy)
{
    const unsigned j = ((unsigned)(jx >> 32) + (1u << 29)) | ((unsigned)(jy >> 32) + (1u << 29));
    unsigned q = 0;
#if defined(__CUDACC__)
#pragma unroll
#endif
    for (int d = 0; d < 9; ++d) q |= (unsigned)(f[d] >> 32) + (1u << 30);
    return ((j | (q >> 1)) >> 30) != 0;
}

}  // namespace plbm
