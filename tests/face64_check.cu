// Host-side check of the lean FP64 face (phd_face64.cuh: states64, hll64) against the plain
// one (face_spatial_f64, temporal, hll_family), compiled for the host: every state and flux
// equal, on seeded random faces -- equal cells, cells equal but for their last bits, smooth
// flow, simple waves, jumps of several decades, near-vacuum rarefactions, cells at rest,
// states that change sign across the face -- with HLL and HLLC, with and without boost, GIZMO
// limiter and slopes, gamma 1.1 to 2.1.  Prints: faces, faces the lean path declined, faces
// that differ.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "phd_ref.cuh"
#include "face64_random.cuh"

using namespace phd;

int main(int argc, char **argv) {
    const long N = argc > 1 ? atol(argv[1]) : 400000;
    std::mt19937_64 rng(20240607);
    long n_open = 0, n_diff = 0;
    RandomFace O;
    for (long t = 0; t < N; t++) {
        random_face(t, rng, O);
        const Face64 &A = O.A;
        const double gamma = O.gamma, dt_half = O.dt_half, *pi = A.pi, *pj = A.pj, *normal = O.normal;
        const bool boost = O.boost, hllc = O.hllc, linear = O.linear, gizmo = O.gizmo;
        const int kind = O.kind;
        double L0[4], R0[4], f0[4], L1[4], R1[4], f1[4];
        if (linear) {
            face_spatial_f64<2>(O.M, 0, 0, 1, pi, pj, A.gi, A.gj, A.w, boost, gizmo, L0, R0);
            temporal<double, 2>(L0, R0, pi, pj, A.gi, A.gj, A.w, gamma, dt_half, boost);
        } else {
            for (int f = 0; f < 4; f++) {
                L0[f] = pi[f] - (boost && (f == 1 || f == 2) ? A.w[f - 1] : 0.);
                R0[f] = pj[f] - (boost && (f == 1 || f == 2) ? A.w[f - 1] : 0.);
            }
        }
        hll_family<double, 2>(hllc, L0, R0, normal, A.w, gamma, boost, f0);
        const Gas64 C = gas64(gamma);
        bool ok = states64(A, C, dt_half, boost, linear, gizmo, L1, R1);
        ok = (hllc ? hll64<true>(L1, R1, normal, A.w, C, boost, f1) : hll64<false>(L1, R1, normal, A.w, C, boost, f1)) && ok;
        if (!ok) { n_open++; continue; }
        bool same = true;
        for (int f = 0; f < 4; f++)
            same = same && L0[f] == L1[f] && R0[f] == R1[f] && (f0[f] == f1[f] || (f0[f] != f0[f] && f1[f] != f1[f]));
        if (!same && n_diff++ < 5)
            fprintf(stderr, "kind %d gamma %g boost %d hllc %d linear %d gizmo %d: %.17g %.17g | %.17g %.17g %.17g %.17g | %.17g %.17g %.17g %.17g\n",
                    kind, gamma, boost, hllc, linear, gizmo, L0[0] - L1[0], R0[0] - R1[0], f0[0], f0[1], f0[2], f0[3], f1[0], f1[1], f1[2], f1[3]);
    }
    printf("%ld %ld %ld\n", N, n_open, n_diff);
    return 0;
}
