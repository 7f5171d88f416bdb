// Compares strict::fast_collide with the plain double sequence of the reference's BGK update, bit for
// bit, on random nodes of one kind.  Usage: strict_test KIND COUNT SEED; prints "compared N of M".
#include "plbm_strict.cuh"

#include <cstdio>
#include <cstdlib>
#include <random>
#include <string>

using namespace plbm::strict;

static void plain(double f[9], double omega, double m[4])
{
    double rho = f[0];
    for (int d = 1; d < 9; ++d) rho = rho + f[d];
    double jx = -f[0] + f[2];
    jx = jx - f[3]; jx = jx + f[5]; jx = jx - f[6]; jx = jx + f[8];
    double jy = -f[0] - f[1];
    jy = jy - f[2]; jy = jy + f[6]; jy = jy + f[7]; jy = jy + f[8];
    const double usq = jx * jx + jy * jy, h = 1.5 * usq;
    const double a[4] = { jx, jy, jx + jy, jx - jy };
    double feq[9];
    feq[4] = (4.0 / 9) * (rho - h);
    for (int k = 0; k < 4; ++k) {
        const double c3 = 3.0 * a[k], c45 = (4.5 * a[k]) * a[k], w = k < 2 ? 1.0 / 9 : 1.0 / 36;
        const int d = k == 0 ? 5 : k == 1 ? 7 : k == 2 ? 8 : 2;
        feq[d] = w * (((rho + c3) + c45) - h);
        feq[8 - d] = w * (((rho - c3) + c45) - h);
    }
    for (int d = 0; d < 9; ++d) f[d] = -omega * (f[d] - feq[d]) + f[d];
    m[0] = rho; m[1] = jx; m[2] = jy; m[3] = usq;
}

int main(int argc, char **argv)
{
    const std::string kind = argc > 1 ? argv[1] : "flow";
    const long count = argc > 2 ? std::atol(argv[2]) : 100000;
    std::mt19937_64 g(argc > 3 ? std::atol(argv[3]) : 1);
    std::uniform_real_distribution<double> u(0, 1);
    std::normal_distribution<double> N(0, 1);
    const double w[9] = { 1.0 / 36, 1.0 / 9, 1.0 / 36, 1.0 / 9, 4.0 / 9, 1.0 / 9, 1.0 / 36, 1.0 / 9, 1.0 / 36 };
    long compared = 0;
    for (long i = 0; i < count; ++i) {
        const double rho = kind == "unit" || kind == "rest" ? 1.0 : 0.8 + 0.6 * u(g);
        double scale = 0.15 * std::pow(10.0, -6 * u(g));
        if (kind == "tiny") scale = 1e-13;
        if (kind == "rest") scale = 0;
        const double jx = scale * N(g), jy = kind == "axis" ? 0 : scale * N(g), noise = std::pow(10.0, -3 - 8 * u(g));
        double f[9], r[9], o[9], m[4];
        for (int d = 0; d < 9; ++d) {
            const double cu = (d % 3 - 1) * jx + (d / 3 - 1) * jy;
            f[d] = w[d] * (rho + 3 * cu + 4.5 * cu * cu - 1.5 * (jx * jx + jy * jy));
            if (kind != "rest" && kind != "unit") f[d] *= 1 + noise * N(g);
            // short significands: sums that are exact or lie half way between two doubles
            if (kind == "short") { const double s = std::ldexp(1.0, 12 + (int)(u(g) * 40)); f[d] = std::nearbyint(f[d] * s) / s; }
            if (kind == "ties") { const double s = std::ldexp(1.0, 50 + (int)(u(g) * 8)); f[d] = std::nearbyint(f[d] * s) / s; }
            if (kind == "wild" && u(g) < 0.05) f[d] *= u(g) < 0.3 ? -1 : u(g) < 0.5 ? 1e300 : 20 * u(g);
            if (kind == "wild" && u(g) < 0.01) f[d] = u(g) < 0.5 ? NAN : INFINITY;
            r[d] = f[d];
        }
        const double omega = 1 / (0.5 + u(g));
        plain(r, omega, m);
        Fixed x;
        if (!fast_collide(f, o, omega, x)) continue;
        ++compared;
        bool same = (double)x.rho * 0x1p-61 == m[0] && (double)x.jx * 0x1p-61 == m[1] && (double)x.jy * 0x1p-61 == m[2] &&
                    x.usq122 * 0x1p-122 == m[3];
        for (int d = 0; d < 9; ++d) same = same && bits_of(o[d]) == bits_of(r[d]);
        if (!same) {
            std::printf("node %ld differs\n", i);
            for (int d = 0; d < 9; ++d) std::printf("  f %a plain %a fixed %a\n", f[d], r[d], o[d]);
            return 1;
        }
    }
    std::printf("compared %ld of %ld\n", compared, count);
    return 0;
}
