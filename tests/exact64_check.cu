// Host-side check of the lean exact flux (phd_exact64.cuh) against the plain one (exact_flux of
// phd_physics.cuh with the host's pow), compiled for the host, on the seeded random faces of
// face64_random.cuh.  Prints: faces, faces the lean path declined, disagreements of the
// convergence flag, the worst difference of a flux component over its scale (rho c, rho c^2,
// rho c^3 of the two sides, at least the component itself), faces beyond 1e-12.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "phd_ref.cuh"
#include "phd_exact64.cuh"
#include "face64_random.cuh"

using namespace phd;

int main(int argc, char **argv) {
    const long N = argc > 1 ? atol(argv[1]) : 400000;
    std::mt19937_64 rng(424242);
    long n_open = 0, n_flag = 0, n_off = 0;
    double worst = 0.;
    RandomFace O;
    for (long t = 0; t < N; t++) {
        random_face(t, rng, O);
        const Face64 &A = O.A;
        double L[4], R[4], f0[4], f1[4];
        for (int f = 0; f < 4; f++) {
            L[f] = A.pi[f] - (f == 1 || f == 2 ? A.w[f - 1] : 0.);
            R[f] = A.pj[f] - (f == 1 || f == 2 ? A.w[f - 1] : 0.);
        }
        bool fa = false, fb = false;
        const bool ok = exact64_flux(L, R, O.normal, A.w, exact64(O.gamma), 200, f1, &fb);
        if (!ok) { n_open++; continue; }
        exact_flux<double, 2>(L, R, O.normal, A.w, O.gamma, 200, f0, &fa);
        if (fa != fb) { n_flag++; continue; }
        if (fa) continue;
        const double rho = std::max(L[0], R[0]), c = std::max(std::sqrt(O.gamma * L[3] / L[0]), std::sqrt(O.gamma * R[3] / R[0])) +
                                                     std::hypot(A.w[0], A.w[1]);
        const double sc[4] = {rho * c, rho * c * c, rho * c * c, rho * c * c * c};
        double r = 0.;
        for (int f = 0; f < 4; f++) r = std::max(r, std::fabs(f0[f] - f1[f]) / std::max(sc[f], std::fabs(f0[f])));
        if (!(r <= 1e-12) && n_off++ < 5) fprintf(stderr, "t %ld kind %d gamma %g r %g\n", t, O.kind, O.gamma, r);
        worst = std::max(worst, r);
    }
    printf("%ld %ld %ld %.3e %ld\n", N, n_open, n_flag, worst, n_off);
    return 0;
}
