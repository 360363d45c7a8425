// Host-side check of the lean reverse of the FP64 face (phd_adjface64.cuh) against the plain
// one (phd_adjoint.cuh: gizmo_pair_adj, temporal_adj, hll_family_adj), compiled for the host,
// on the seeded random faces of face64_random.cuh with random output weights: the 24 adjoints
// of the cells' values and slopes.  The two take the same branches and differ in rounding
// alone, so the difference is taken against the largest term each adjoint is summed from
// (the plain reverse of the absolute chain is not available, so: of the largest adjoint of
// its kind, scaled by the field).  Prints: faces, faces the lean path declined, the worst
// relative difference, faces beyond 1e-9, and by the median face the difference in units of
// 2^-53.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "phd_ref.cuh"
#include "phd_adjoint.cuh"
#include "phd_adjface64.cuh"
#include "face64_random.cuh"

using namespace phd;

int main(int argc, char **argv) {
    const long N = argc > 1 ? atol(argv[1]) : 400000;
    std::mt19937_64 rng(20240607);
    std::normal_distribution<double> G(0., 1.);
    long n_open = 0, n_off = 0;
    double worst = 0.;
    std::vector<double> all;
    RandomFace O;
    for (long t = 0; t < N; t++) {
        random_face(t, rng, O);
        const Face64 &A = O.A;
        const double gamma = O.gamma, dt = O.dt_half, *pi = A.pi, *pj = A.pj, c = O.c;
        const bool boost = O.boost, gizmo = O.gizmo, linear = O.linear;
        // weights that make each flux component count alike
        const double aF[4] = {G(rng) / (pi[0] * c), G(rng) / (pi[0] * c * c), G(rng) / (pi[0] * c * c),
                              G(rng) / (pi[0] * c * c * c)};
        double want[24] = {0.}, got[24] = {0.};
        {   // plain
            double sl[4], sr[4], L0[4], R0[4], Ls[4], Rs[4], L[4], R[4];
            for (int f = 0; f < 4; f++) {
                sl[f] = pi[f] - (boost && (f == 1 || f == 2) ? A.w[f - 1] : 0.);
                sr[f] = pj[f] - (boost && (f == 1 || f == 2) ? A.w[f - 1] : 0.);
                L0[f] = sl[f];
                R0[f] = sr[f];
            }
            double si[2], sj[2], mi = 0., mj = 0., md = 0.;
            for (int k = 0; k < 2; k++) {
                si[k] = A.com[k] - (A.xi[k] + A.ci[k]);
                sj[k] = A.com[k] - (A.xj[k] + A.cj[k]);
                mi += si[k] * si[k];
                mj += sj[k] * sj[k];
                md += (A.xj[k] - A.xi[k]) * (A.xj[k] - A.xi[k]);
                for (int f = 0; f < 4 && linear; f++) {
                    L0[f] = L0[f] + A.gi[2 * f + k] * si[k];
                    R0[f] = R0[f] + A.gj[2 * f + k] * sj[k];
                }
            }
            mi = std::sqrt(mi); mj = std::sqrt(mj); md = std::sqrt(md);
            bool rl = false, rr = false;
            for (int f = 0; f < 4; f++) { Ls[f] = L0[f]; Rs[f] = R0[f]; }
            if (linear && gizmo) {
                for (int f = 0; f < 4; f++) gizmo_pair<double>(sl[f], sr[f], pi[f], pj[f], mi, mj, md, Ls[f], Rs[f]);
                rl = Ls[0] < 0. || Ls[3] < 0.;
                rr = Rs[0] < 0. || Rs[3] < 0.;
                for (int f = 0; f < 4; f++) { if (rl) Ls[f] = sl[f]; if (rr) Rs[f] = sr[f]; }
            }
            for (int f = 0; f < 4; f++) { L[f] = Ls[f]; R[f] = Rs[f]; }
            if (linear) temporal<double, 2>(L, R, pi, pj, A.gi, A.gj, A.w, gamma, dt, boost);
            double aL[4] = {0.}, aR[4] = {0.}, aLs[4] = {0.}, aRs[4] = {0.};
            hll_family_adj<double>(O.hllc, L, R, O.normal, A.w, gamma, boost, aF, aL, aR);
            double *api = want, *apj = want + 4, *agi = want + 8, *agj = want + 16;
            if (linear) {
                temporal_adj<double>(Ls, Rs, pi, pj, A.gi, A.gj, A.w, gamma, dt, boost, aL, aR, aLs, aRs, api, apj, agi, agj);
                for (int f = 0; f < 4; f++) {
                    double as = 0., bs = 0., ax = 0., bx = 0.;
                    if (gizmo) {
                        if (rl) as += aLs[f];
                        if (rr) bs += aRs[f];
                        gizmo_pair_adj<double>(sl[f], sr[f], pi[f], pj[f], mi, mj, md, L0[f], R0[f], rl ? 0. : aLs[f],
                                               rr ? 0. : aRs[f], as, bs, ax, bx);
                    } else {
                        ax = aLs[f];
                        bx = aRs[f];
                    }
                    for (int k = 0; k < 2; k++) { agi[2 * f + k] += ax * si[k]; agj[2 * f + k] += bx * sj[k]; }
                    api[f] += as + ax;
                    apj[f] += bs + bx;
                }
            } else {
                for (int f = 0; f < 4; f++) { api[f] = aL[f]; apj[f] = aR[f]; }
            }
        }
        const Gas64 C = gas64(gamma);
        double sl[4], sr[4], L[4], R[4], aL[4] = {0.}, aR[4] = {0.};
        StateDecisions D;
        bool ok = linear ? states64_decide(A, C, dt, boost, gizmo, sl, sr, L, R, D)
                         : states64(A, C, dt, boost, false, false, L, R);
        ok = ok && (O.hllc ? hll64_adj<true>(L, R, O.normal, A.w, C, boost, aF, aL, aR)
                           : hll64_adj<false>(L, R, O.normal, A.w, C, boost, aF, aL, aR));
        if (ok && linear) {
            double asl[4], aol[4], asr[4], aor[4], rl, pl, rr, pr;
            side64_rev(aL, D.half_l, D.spat_l, gizmo, false, D, pi, A.gi, sl, sr, gamma, dt, asl, aol, got + 8, rl, pl, ok);
            side64_rev(aR, D.half_r, D.spat_r, gizmo, true, D, pj, A.gj, sr, sl, gamma, dt, asr, aor, got + 16, rr, pr, ok);
            for (int f = 0; f < 4; f++) {
                got[f] = asl[f] + aor[f] + (f == 0 ? rl : (f == 3 ? pl : 0.));
                got[4 + f] = asr[f] + aol[f] + (f == 0 ? rr : (f == 3 ? pr : 0.));
            }
        } else if (ok) {
            for (int f = 0; f < 4; f++) { got[f] = aL[f]; got[4 + f] = aR[f]; }
        }
        if (!ok) { n_open++; continue; }
        // each adjoint times its variable's scale (rho, c, c, p; slopes over the cell's size)
        const double sc[4] = {std::max(pi[0], pj[0]), c, c, std::max(pi[3], pj[3])};
        double big = 0., off = 0.;
        for (int q = 0; q < 24; q++) {
            const double s = q < 8 ? sc[q % 4] : sc[((q - 8) / 2) % 4] / O.h;
            big = std::max(big, std::fabs(want[q]) * s);
            off = std::max(off, std::fabs(want[q] - got[q]) * s);
        }
        const double r = big > 0. ? off / big : off;
        if (!(r <= 1e-9) && n_off++ < 5)
            fprintf(stderr, "t %ld kind %d hllc %d boost %d linear %d gizmo %d r %g\n", t, O.kind, O.hllc, boost, linear, gizmo, r);
        worst = std::max(worst, r);
        all.push_back(r);
    }
    std::nth_element(all.begin(), all.begin() + all.size() / 2, all.end());
    printf("%ld %ld %.3e %ld %.2f\n", N, n_open, worst, n_off, all[all.size() / 2] * 9007199254740992.);
    return 0;
}
