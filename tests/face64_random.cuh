// Seeded random faces for the host checks of the lean FP64 face and its reverse: equal cells,
// cells equal but for their last bits, smooth flow, simple waves, jumps of several decades,
// near-vacuum rarefactions, states that change sign across the face, supersonic flow; cells
// at rest and with zero slopes among them; gamma 1.1 to 2.1.
#pragma once
#include <cmath>
#include <random>

#include "phd_face64.cuh"

struct RandomFace {
    phd::Face64 A;
    double gamma, c, h, dt_half, x[4], dcom[4], com[2], vol[2], area, normal[2];
    bool boost, hllc, linear, gizmo;
    int kind;
    phd_mesh M;
};

inline void random_face(long t, std::mt19937_64 &rng, RandomFace &O) {
    using phd::Face64;
    std::uniform_real_distribution<double> U(0., 1.);
    auto S = [&](double a) { return a * (2. * U(rng) - 1.); };
    Face64 &A = O.A;
    double *x = O.x, *dcom = O.dcom, *com = O.com, *normal = O.normal;
    const double gamma = O.gamma = (t % 3 == 0) ? 1.4 : (t % 3 == 1 ? 5. / 3. : 1.1 + U(rng));
    const int kind = O.kind = int((t / 3) % 8);
    O.boost = U(rng) < 0.7;
    O.hllc = U(rng) < 0.6;
    O.linear = U(rng) < 0.85;
    O.gizmo = U(rng) < 0.8;
    const double h = O.h = std::exp(S(4.)), angle = S(3.14159);
    O.vol[0] = O.vol[1] = h * h;
    O.area = h;
    normal[0] = std::cos(angle);
    normal[1] = std::sin(angle);
    x[0] = S(1.); x[2] = S(1.);
    x[1] = x[0] + h * normal[0]; x[3] = x[2] + h * normal[1];
    const double off = S(0.3);
    com[0] = 0.5 * (x[0] + x[1]) - off * h * normal[1];
    com[1] = 0.5 * (x[2] + x[3]) + off * h * normal[0];
    for (int k = 0; k < 4; k++) dcom[k] = (t % 5 == 0) ? 0. : S(0.1 * h);
    double *pi = A.pi, *pj = A.pj;
    pi[0] = std::exp(S(2.)); pi[3] = std::exp(S(2.));
    const double c = O.c = std::sqrt(gamma * pi[3] / pi[0]);
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
    O.dt_half = 0.1 * h / (c + 1e-3);
    O.M = phd_mesh{};
    O.M.dim = 2; O.M.n_cells = 2; O.M.n_real = 2; O.M.n_faces = 1;
    O.M.x = x; O.M.dcom = dcom; O.M.vol = O.vol; O.M.com = com; O.M.area = &O.area; O.M.normal = normal;
}
