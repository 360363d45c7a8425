// Host-side check of the fixed-point powers (phd_fp64.cuh: log2_fix, exp2_fix) against the
// 80-bit powl, compiled for the host: seeded bases within 2^-40 of 1, around 1, over 30 and
// over 600 binades, exponents of the exact Riemann solver for gamma in (1.05, 3).  Prints:
// powers, the largest error in units of the last place, powers not correctly rounded, powers
// of 1 that are not 1, declined.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "phd_fp64.cuh"

using namespace phd;

int main(int argc, char **argv) {
    const long N = argc > 1 ? atol(argv[1]) : 1000000;
    std::mt19937_64 rng(77);
    std::uniform_real_distribution<double> U(0., 1.);
    long n_bad = 0, n_one = 0, n_open = 0;
    double worst = 0.;
    for (long t = 0; t < N; t++) {
        const double g = t % 3 == 0 ? 1.4 : (t % 3 == 1 ? 5. / 3. : 1.05 + 1.95 * U(rng));
        const double ys[6] = {(g - 1.) / (2. * g), -(g + 1.) / (2. * g), 1. / g, 2. / (g - 1.), 2. * g / (g - 1.),
                              0.01 + 15. * U(rng)};
        const double y = ys[t % 6];
        const int kind = (int)((t / 18) % 4);
        double x = 1. + (2. * U(rng) - 1.) * std::ldexp(1., -(int)(40. * U(rng)) - 1);
        if (kind == 1) x = 0.25 + 4. * U(rng);
        if (kind == 2) x = std::exp2(30. * (U(rng) - 0.5));
        if (kind == 3) x = std::exp2(600. * (U(rng) - 0.5));
        bool ok = log2_ok(x);
        const double p = exp2_fix(log2_fix(x), y, ok);
        if (!ok) { n_open++; continue; }
        const long double want = powl((long double)x, (long double)y);
        const double ulp = std::nextafter(std::fabs(p), INFINITY) - std::fabs(p);
        worst = std::fmax(worst, (double)(fabsl((long double)p - want) / ulp));
        if ((double)want != p) n_bad++;
        ok = true;
        if (exp2_fix(log2_fix(1.0), y, ok) != 1.0 || !ok) n_one++;
    }
    printf("%ld %.4f %ld %ld %ld\n", N, worst, n_bad, n_one, n_open);
    return 0;
}
