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
#include "phd_face64.cuh"

using namespace phd;

int main(int argc, char **argv) {
    const long N = argc > 1 ? atol(argv[1]) : 400000;
    std::mt19937_64 rng(20240607);
    std::uniform_real_distribution<double> U(0., 1.);
    auto S = [&](double a) { return a * (2. * U(rng) - 1.); };
    long n_open = 0, n_diff = 0;
    for (long t = 0; t < N; t++) {
        const double gamma = (t % 3 == 0) ? 1.4 : (t % 3 == 1 ? 5. / 3. : 1.1 + U(rng));
        const int kind = int((t / 3) % 8);
        const bool boost = U(rng) < 0.7, hllc = U(rng) < 0.6, linear = U(rng) < 0.85, gizmo = U(rng) < 0.8;
        const double h = std::exp(S(4.)), angle = S(3.14159);
        double x[4], dcom[4], com[2], vol[2] = {h * h, h * h}, area = h, normal[2] = {std::cos(angle), std::sin(angle)};
        x[0] = S(1.); x[2] = S(1.);
        x[1] = x[0] + h * normal[0]; x[3] = x[2] + h * normal[1];
        const double off = S(0.3);
        com[0] = 0.5 * (x[0] + x[1]) - off * h * normal[1];
        com[1] = 0.5 * (x[2] + x[3]) + off * h * normal[0];
        for (int k = 0; k < 4; k++) dcom[k] = (t % 5 == 0) ? 0. : S(0.1 * h);
        Face64 A;
        double *pi = A.pi, *pj = A.pj;
        pi[0] = std::exp(S(2.)); pi[3] = std::exp(S(2.));
        const double c = std::sqrt(gamma * pi[3] / pi[0]);
        pi[1] = (t % 7 == 0) ? 0. : S(2. * c); pi[2] = (t % 7 == 0) ? 0. : S(2. * c);
        for (int f = 0; f < 4; f++) pj[f] = pi[f];
        double amp = 0.;
        if (kind == 1) {                               // the last bits
            for (int f = 0; f < 4; f++) pj[f] *= 1. + 2.220446049250313e-16 * std::floor(S(4.));
        } else if (kind == 2) {                        // smooth
            amp = std::pow(10., -8. * U(rng));
            for (int f = 0; f < 4; f++) pj[f] += (f == 1 || f == 2 ? c : pi[f]) * S(amp);
        } else if (kind == 3) {                        // simple wave: u - 2c/(g-1) or u + 2c/(g-1) kept
            amp = std::pow(10., -6. * U(rng));
            const double k = std::exp(S(amp)), cj = c * std::pow(k, 0.5 * (gamma - 1.) / gamma);
            pj[3] *= k;
            pj[0] *= std::pow(k, 1. / gamma);
            const double du = (U(rng) < 0.5 ? 2. : -2.) * (cj - c) / (gamma - 1.);
            pj[1] += du * normal[0]; pj[2] += du * normal[1];
        } else if (kind == 4) {                        // jumps
            pj[0] = std::exp(S(5.)); pj[3] = std::exp(S(8.));
            pj[1] = S(3.); pj[2] = S(3.);
        } else if (kind == 5) {                        // strong rarefaction
            const double du = (2. + 10. * U(rng)) * c * U(rng);
            pj[1] += du * normal[0]; pj[2] += du * normal[1];
        } else if (kind == 6) {                        // sign changes
            for (int f = 1; f < 3; f++) { pi[f] = S(1e-3); pj[f] = S(1e-3); }
            pj[0] *= 1. + S(0.1);
            pj[3] *= 1. + S(0.1);
        } else if (kind == 7) {                        // supersonic
            pi[1] += 4. * c * normal[0]; pi[2] += 4. * c * normal[1];
            pj[1] = pi[1] + S(0.1 * c); pj[2] = pi[2]; pj[3] *= 1. + S(0.2);
        }
        if (t % 11 == 0) for (int k = 0; k < 2; k++) { pi[1 + k] = -pi[1 + k]; pj[1 + k] = -pj[1 + k]; }
        const double ga = (kind == 0 && t % 2) ? 0. : (t % 13 == 0 ? 3. : 0.5) * (amp > 0. ? amp : 0.1) / h;
        for (int f = 0; f < 4; f++)
            for (int k = 0; k < 2; k++) {
                const double s = (f == 1 || f == 2) ? c : pi[f];
                A.gi[2 * f + k] = S(ga * s);
                A.gj[2 * f + k] = S(ga * s);
            }
        const bool still = t % 6 == 0;
        for (int k = 0; k < 2; k++) {
            A.w[k] = still ? 0. : 0.5 * (pi[1 + k] + pj[1 + k]) + S(1e-3 * c);
            A.xi[k] = x[2 * k]; A.xj[k] = x[2 * k + 1];
            A.ci[k] = dcom[2 * k]; A.cj[k] = dcom[2 * k + 1];
            A.com[k] = com[k];
        }
        const double dt_half = 0.1 * h / (c + 1e-3);
        phd_mesh M = {};
        M.dim = 2; M.n_cells = 2; M.n_real = 2; M.n_faces = 1;
        M.x = x; M.dcom = dcom; M.vol = vol; M.com = com; M.area = &area; M.normal = normal;
        double L0[4], R0[4], f0[4], L1[4], R1[4], f1[4];
        if (linear) {
            face_spatial_f64<2>(M, 0, 0, 1, pi, pj, A.gi, A.gj, A.w, boost, gizmo, L0, R0);
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
