// Compares the products and the relaxation of the F64_Q60 collision with a plain formulation, bit for bit, on random
// and on edge values: high words of three 32 x 32-bit products of the unsigned bit patterns, corrected afterwards for
// negative factors.  Usage: q60_test COUNT SEED; prints "compared N".
#include "plbm_consts.h"
#include "plbm_q60.cuh"

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

typedef unsigned long long u64;
typedef long long i64;
typedef unsigned __int128 u128;

static u64 high(u64 a, u64 b)
{
    const u64 m = 0xffffffffull, al = a & m, ah = a >> 32, bl = b & m, bh = b >> 32;
    return (u64)((u128)ah * bh + (u128)(ah * bl >> 32) + (u128)(al * bh >> 32));
}
static i64 by_constant(u64 c, i64 v) { return (i64)(high(c, (u64)v) - (v < 0 ? c : 0)); }
static i64 by_value(i64 a, i64 b)
{
    const u64 x = (u64)a << 2, y = (u64)b << 2;
    return (i64)(high(x, y) - ((i64)x < 0 ? y : 0) - ((i64)y < 0 ? x : 0));
}
static void relax(i64 f[9], i64 jx, i64 jy, i64 jx2, i64 jy2, i64 jxy, i64 R, const plbm::StepParams &p)
{
    const u64 w = (u64)p.q_om1;
    const i64 usq = jx2 + jy2, b9 = by_constant((u64)p.q_ow9, R), b36 = by_constant((u64)p.q_ow36, R);
    f[4] = f[4] + by_constant((u64)p.q_ow49, R) - 2 * by_constant(w, f[4]);
    const i64 u[4] = { jx, jy, jx + jy, jx - jy }, u2[4] = { jx2, jy2, usq + 2 * jxy, usq - 2 * jxy };
    const int plus[4] = { 5, 7, 8, 2 };
    for (int k = 0; k < 4; ++k) {
        const i64 sym = by_constant((u64)(k < 2 ? p.q_k9 : p.q_k36), u2[k]) + (k < 2 ? b9 : b36);
        const i64 odd = by_constant((u64)(k < 2 ? p.q_o9 : p.q_o36), u[k]);
        const int d = plus[k];
        f[d] = f[d] + sym + odd - 2 * by_constant(w, f[d]);
        f[8 - d] = f[8 - d] + sym - odd - 2 * by_constant(w, f[8 - d]);
    }
}

static long bad = 0;
static void check(bool same, const char *what, i64 a, i64 b)
{
    if (!same && ++bad < 10) std::printf("%s differs at %lld, %lld\n", what, a, b);
}

int main(int argc, char **argv)
{
    const long count = argc > 1 ? std::atol(argv[1]) : 100000;
    std::mt19937_64 g(argc > 2 ? std::atol(argv[2]) : 1);
    const i64 one = 1ll << 60;
    // zero, one unit, low words with bit 31 alone and full, the ends of [-2, 2) and [-4, 4)
    const i64 edges[] = { 0, 1, -1, 1ll << 31, -(1ll << 31), (1ll << 31) - 1, 0xffffffffll, -0xffffffffll, (1ll << 32), one, -one,
                          2 * one - 1, -2 * one, -2 * one + 1, one | 0x80000000ll, -(one | 0x80000000ll), 4 * (one - 1) + 3,
                          -4 * one, one / 2, -one / 2, one + 0x7fffffff };
    const int n = sizeof edges / sizeof *edges;
    long compared = 0;
    auto pick = [&](int shift) -> i64 { return g() % 4 == 0 ? edges[g() % n] : (i64)g() >> shift; };
    auto products = [&](u64 c, i64 a, i64 b) {
        check(plbm::mulc(c, a) == by_constant(c, a), "mulc", (i64)c, a);
        if (a >= 0) check(plbm::mulc<true>(c, a) == by_constant(c, a), "mulc<true>", (i64)c, a);
        const u64 h = c >> 2;   // below 1/4
        check(plbm::mulc_half(h, a) == by_constant(h, a), "mulc_half", (i64)h, a);
        check(plbm::mulv(a, b) == by_value(a, b), "mulv", a, b);
        ++compared;
    };
    for (int i = 0; i < n; ++i)
        for (int j = 0; j < n; ++j)
            for (u64 c : { 0ull, 1ull, 1ull << 31, 1ull << 32, 0xffffffffull, ~0ull, ~0ull << 31, (u64)edges[j] })
                products(c, edges[i], edges[j]);
    plbm::StepParams p;
    std::memset(&p, 0, sizeof p);
    for (long k = 0; k < count; ++k) {
        products(g() >> (g() % 3), pick(1 + g() % 30), pick(1 + g() % 30));
        if (k % 1000 == 0) {
            p.omega = 1 / (0.501 + 2.0 * (double)(g() % 1000) / 1000);
            p.rho_out = 1;
            plbm::fill_q60_constants(p);
        }
        // a node: populations about the rest state, some of any size and sign
        i64 f[9], want[9], a[9], b[9];
        const bool wild = g() % 3 == 0;
        for (int d = 0; d < 9; ++d)
            f[d] = wild ? pick(2 + g() % 8) : plbm::q60((d == 4 ? 4.0 / 9 : d % 2 ? 1.0 / 9 : 1.0 / 36) * (0.7 + 0.6 * (double)(g() >> 11) * 0x1p-53));
        const i64 jx = f[2] + f[5] + f[8] - (f[0] + f[3] + f[6]), jy = f[6] + f[7] + f[8] - (f[0] + f[1] + f[2]);
        i64 rho = 0;
        for (int d = 0; d < 9; ++d) rho += f[d];
        bool out = jx >= 2 * one || jx < -2 * one || jy >= 2 * one || jy < -2 * one;
        for (int d = 0; d < 9; ++d) out = out || f[d] >= 4 * (one - 1) + 4 || f[d] < -4 * one;
        check(plbm::q60_out_of_range(f, jx, jy) == out, "range", jx, jy);
        if (out) continue;
        const i64 jx2 = by_value(jx, jx), jy2 = by_value(jy, jy), jxy = by_value(jx, jy), usq = jx2 + jy2, R = rho - (usq + (usq >> 1));
        bool positive = R >= 0;
        for (int d = 0; d < 9; ++d) { want[d] = a[d] = b[d] = f[d]; positive = positive && f[d] >= 0; }
        relax(want, jx, jy, jx2, jy2, jxy, R, p);
        plbm::relax_q60<false>(a, jx, jy, jx2, jy2, jxy, R, p);
        for (int d = 0; d < 9; ++d) check(a[d] == want[d], "relax_q60<false>", a[d], want[d]);
        if (!positive) continue;
        plbm::relax_q60<true>(b, jx, jy, jx2, jy2, jxy, R, p);
        for (int d = 0; d < 9; ++d) check(b[d] == want[d], "relax_q60<true>", b[d], want[d]);
        compared += 1;
    }
    std::printf("compared %ld\n", compared);
    return bad ? 1 : 0;
}
