// phd_face64.cuh -- one face of the FP64 path with as few FP64 instructions as its results need.
//
// The same numbers as face_spatial_f64 + temporal + hll_family (phd_ref.cuh, phd_physics.cuh),
// bit for bit: every product and sum that is rounded there is rounded here, in the same
// order.  What differs is the work around them (phd_fp64.cuh tells why it matters):
//   * quotients and roots from FP32 / integer seeds, the quotients of one denominator
//     sharing its seed;
//   * comparisons, minima, maxima and sign tests on the bits; factors 1/2 and 1/4 are
//     exact and ride in a fused multiply-add with the addition that follows them;
//   * the star state is formed once, for the side of the contact it lies on;
//   * the two-rarefaction pressure (three powers, 250 FP64 instructions for a warp in which
//     one face takes it) only decides whether it exceeds the sides' pressures: where an
//     FP32 estimate with a margin for its rounding settles that (trrs_below), the wave
//     speeds are those of two rarefactions and the pressure is not formed.
// A face whose operands leave the windows in which this holds (infinities, NaN, magnitudes
// beyond 2^80, vanishing denominators) returns false and takes the plain path.
#pragma once
#include "phd_fp64.cuh"
#include "phd_physics.cuh"

namespace phd {

// Constants of gamma, formed once on the host with the operations the plain path repeats.
struct Gas64 {
    double g, gm1, y_gm1;              // gamma, gamma - 1 and the reciprocal seed of the latter
    double gp1, gm1_gp1, gp1_2g;       // gamma + 1, (g-1)/(g+1), (g+1)/(2g)
    float zf, half_gm1f;               // (g-1)/(2g), (g-1)/2
    int ok;                            // gamma - 1 and gamma + 1 within the seeds' window
};

inline Gas64 gas64(double gamma) {
    Gas64 C;
    C.g = gamma;
    C.gm1 = gamma - 1.0;
    C.y_gm1 = 1.0 / C.gm1;
    C.gp1 = gamma + 1.0;
    C.gm1_gp1 = C.gm1 / C.gp1;
    C.gp1_2g = C.gp1 / (2.0 * gamma);
    C.zf = (float)(C.gm1 / (2.0 * gamma));
    C.half_gm1f = (float)(0.5 * C.gm1);
    C.ok = C.gm1 > 1e-3 && C.gm1 < 1e3;
    return C;
}

// Whether the two-rarefaction pressure p* lies at or below both sides' pressures, decided in
// FP32.  p* is the root of F(p) = f_L + f_R + (u_R - u_L), f_K = 2 c_K/(g-1) ((p/p_K)^z - 1),
// so it is below p_min exactly when F(p_min) > 0: with c_M the sound speed on the side of
// p_max, when G = (g-1)/2 (u_R - u_L) / c_M exceeds X = 1 - (p_min/p_max)^z.  true only
// when that holds by more than the FP32 rounding of both sides (1e-6 each) and the FP64
// rounding of the plain path's own p*, and the powers' bases are positive (no vacuum).
PHD_HD __forceinline__ bool trrs_below(double dp, double p_max, double du, double cm, double c_sum, double ul,
                                       double ur, const Gas64 &C) {
    // FP32's exponents must hold p_max, the differences down to its last bit, and the speeds
    if (f64_hi(p_max) - ((1023u - 60u) << 20) >= (180u << 20) || f64_hi(c_sum) - ((1023u - 60u) << 20) >= (160u << 20))
        return false;
    const float d = f64_to_f32(dp) / f64_to_f32(p_max);
    const float cs = f64_to_f32(c_sum), g = -C.half_gm1f * f64_to_f32(du);     // (g-1)/2 (u_R - u_L)
    const float cmf = f64_to_f32(cm);
    const float X = -expm1f(C.zf * log1pf(-d));
    const float noise = 1e-12f * (cs + fabsf(f64_to_f32(ul)) + fabsf(f64_to_f32(ur)));
    return d < 0.9f && cs - g > 1e-3f * cs && g * (1.f - 4e-6f) - X * cmf * (1.f + 4e-6f) > noise;
}

// The plain two-rarefaction pressure (get_waves), for the faces that trrs_below leaves open.
#ifdef __CUDACC__
__host__ __device__ __noinline__
#endif
inline double trrs_pressure(double ul, double pl, double cl, double ur, double pr, double cr, double gamma) {
    const double z = (gamma - 1.) / (2. * gamma);
    const double plr = pow(pl / pr, z);
    const double u_star = ((((plr * ul) / cl) + (ur / cr)) + ((2. * (plr - 1.)) / (gamma - 1.))) /
                          ((plr / cl) + (1. / cr));
    double p = (.5 * pl) * pow((1. + (((gamma - 1.) * (ul - u_star)) / (2. * cl))), (1. / z));
    return p + ((.5 * pr) * pow((1. + (((gamma - 1.) * (u_star - ur)) / (2. * cr))), (1. / z)));
}

// get_waves: wave speeds, and m = d (s - u) of both sides (the contact speed's terms, which
// the star state uses again).
PHD_HD __forceinline__ bool waves64(double dl, double ul, double pl, double dr, double ur, double pr, const Gas64 &C,
                                    double &sl, double &sc, double &sr, double &ml, double &mr) {
    bool ok = f64_pos(pl) && f64_pos(pr);
    const double cl = f64_sqrt(f64_div(C.g * pl, dl, ok), ok), cr = f64_sqrt(f64_div(C.g * pr, dr, ok), ok);
    ok = ok && f64_lt(1.0E-10, cl) && f64_lt(1.0E-10, cr);
    const double cs = cl + cr, du = ul - ur;
    // (pl + pr)/2 + (du/2) ((dl + dr)/2) ((cl + cr)/2), its powers of two taken together
    const double pv = f64_half(fma(0.25, (du * (dl + dr)) * cs, pl + pr), ok);
    double ps = f64_neg(pv) ? 0. : pv;
    const long long kl = f64_key(pl), kr = f64_key(pr), ks = f64_key(ps);
    const bool lr = kl <= kr;
    const double p_min = lr ? pl : pr, p_max = lr ? pr : pl;
    const long long kmin = lr ? kl : kr, kmax = lr ? kr : kl;
    bool shocks = true;
    // p_max / p_min < 2 as p_max < 2 p_min (the same for positive pressures: a quotient that
    // is below 2 is at most 2 - 2^-52)
    if (kmax < kmin + (1ll << 52) && kmin < ks && ks < kmax) {
    } else if (ks <= kmin) {
        const double dp = p_max - p_min;
        // equal states: the plain path's p* is p itself (its u* is within 3 ulp of u, and
        // (g-1)/2 |u|/c 3 ulp < 2^-54 leaves the powers' bases at 1)
        const bool same = f64_zero(dp) && f64_zero(du) && f64_bits(dl) == f64_bits(dr) &&
                          C.half_gm1f * fabsf(f64_to_f32(ul)) < 0.15f * f64_to_f32(cl);
        if (same || trrs_below(dp, p_max, du, lr ? cr : cl, cs, ul, ur, C)) shocks = false;
        else {
            ps = trrs_pressure(ul, pl, cl, ur, pr, cr, C.g);
            ok = ok && (f64_hi(ps) & 0x7ff00000u) != 0x7ff00000u;       // a vacuum: no pressure
        }
    } else {
        const double gl = f64_sqrt(f64_div(f64_div(2., C.gp1 * dl, ok), ps + pl * C.gm1_gp1, ok), ok);
        const double gr = f64_sqrt(f64_div(f64_div(2., C.gp1 * dr, ok), ps + pr * C.gm1_gp1, ok), ok);
        ps = f64_div((gl * pl + gr * pr) + du, gl + gr, ok);
    }
    const bool shl = shocks && !(f64_key(ps) <= kl), shr = shocks && !(f64_key(ps) <= kr);
    double al = cl, ar = cr;
    if (shl) al = cl * f64_sqrt(1. + C.gp1_2g * (f64_div(ps, pl, ok) - 1.), ok);
    if (shr) ar = cr * f64_sqrt(1. + C.gp1_2g * (f64_div(ps, pr, ok) - 1.), ok);
    sl = ul - al;
    sr = ur + ar;
    const double bl = sl - ul, br = sr - ur;
    ml = dl * bl;
    mr = dr * br;
    sc = f64_div(((pr - pl) + (dl * ul) * bl) - (dr * ur) * br, ml - mr, ok);
    return ok;
}

// hll_family: HLL / HLLC flux and deboost.
template <bool HLLC>
PHD_HD __forceinline__ bool hll64(const double *L, const double *R, const double *n, const double *w, const Gas64 &C,
                                  bool boost, double *f) {
    const double _dl = L[0], _pl = L[3], _dr = R[0], _pr = R[3];
    const double Vnl = L[1] * n[0] + L[2] * n[1], Vnr = R[1] * n[0] + R[2] * n[1];
    const double wn = boost ? 0. : w[0] * n[0] + w[1] * n[1];
    double sl, sc, sr, ml, mr;
    bool ok = waves64(_dl, Vnl, _pl, _dr, Vnr, _pr, C, sl, sc, sr, ml, mr);
    const bool data_l = f64_le(wn, sl), data_r = !data_l && !f64_le(wn, sr);
    if (HLLC || data_l || data_r) {
        const bool left = data_l || (!data_r && f64_le(wn, sc));
        const double d = left ? _dl : _dr, p = left ? _pl : _pr, Vn = left ? Vnl : Vnr;
        const double v0 = left ? L[1] : R[1], v1 = left ? L[2] : R[2];
        const double e = fma(0.5, d * (v0 * v0 + v1 * v1), f64_div_by(p, C.gm1, C.y_gm1, ok));
        if (data_l || data_r) {
            const double u = boost ? Vn : Vn - wn;
            f[0] = d * u;
            f[3] = e * u + p * Vn;
            f[1] = (d * v0) * u + p * n[0];
            f[2] = (d * v1) * u + p * n[1];
        } else {
            const double s = left ? sl : sr, m = left ? ml : mr;
            const double sw = boost ? s : s - wn;
            const double f1 = f64_div(m, s - sc, ok) * sw, q = sc - Vn;      // factor_1 (s - w.n)
            const double f2 = f1 * q + p, frho = f1 - m;
            f[0] = frho;
            f[3] = ((e + p) * Vn - s * e) + f1 * (f64_div(e, d, ok) + q * (sc + f64_div(p, m, ok)));
            f[1] = frho * v0 + f2 * n[0];
            f[2] = frho * v1 + f2 * n[1];
        }
    } else {
        const double fac1 = boost ? sr : sr - wn, fac2 = boost ? sl : sl - wn, fac3 = sr - sl;
        const double y = f64_rcp(fac3, ok);
        const double el = fma(0.5, _dl * (L[1] * L[1] + L[2] * L[2]), f64_div_by(_pl, C.gm1, C.y_gm1, ok));
        const double er = fma(0.5, _dr * (R[1] * R[1] + R[2] * R[2]), f64_div_by(_pr, C.gm1, C.y_gm1, ok));
        f[0] = f64_div_by((((_dl * Vnl) * fac1 - (_dr * Vnr) * fac2) - (sl * _dl) * fac1) + (sr * _dr) * fac2, fac3, y,
                          ok);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const double kl = _dl * L[1 + k], kr = _dr * R[1 + k];
            f[1 + k] = f64_div_by((((kl * Vnl + _pl * n[k]) * fac1 - (kr * Vnr + _pr * n[k]) * fac2) - (sl * kl) * fac1) +
                                      (sr * kr) * fac2, fac3, y, ok);
        }
        f[3] = f64_div_by(((((el + _pl) * Vnl) * fac1 - ((er + _pr) * Vnr) * fac2) - (sl * el) * fac1) +
                              (sr * er) * fac2, fac3, y, ok);
    }
    if (boost) {
        // deboost, w f_0 formed once
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const double wf = w[k] * f[0];
            f[3] = f[3] + w[k] * fma(0.5, wf, f[1 + k]);
            f[1 + k] = f[1 + k] + wf;
        }
    }
    return ok;
}

// gizmo_pair of one field; qi, qj the centroid distances over the cells' distance.  A bound
// that would change its state's sign (the quotient form) clears ok.
PHD_HD __forceinline__ void gizmo64(double sl, double sr, double ci, double cj, double qi, double qj, double &xl,
                                    double &xr, bool &ok) {
    const long long ki = f64_key(ci), kj = f64_key(cj);
    const double d = sr - sl, ad = f64_from(f64_bits(d) & 0x7fffffffffffffffll);
    const bool up = ki < kj;
    const bool lmin = !(f64_key(sr) < f64_key(sl));
    const double phi_max = lmin ? sr : sl, phi_min = lmin ? sl : sr;
    const double plus = fma(0.5, ad, phi_max), minus = fma(-0.5, ad, phi_min);
    // phi + delta of phi's own sign (or either zero)
    const bool pz = f64_zero(plus) || f64_zero(phi_max) || ((f64_bits(plus) ^ f64_bits(phi_max)) >= 0);
    const bool mz = f64_zero(minus) || f64_zero(phi_min) || ((f64_bits(minus) ^ f64_bits(phi_min)) >= 0);
    double bp = plus, bm = minus;
    const bool same = ki == kj;
    if (!pz && !same) bp = f64_div(phi_max, 1. + f64_div(f64_half(ad, ok), f64_from(f64_bits(phi_max) & 0x7fffffffffffffffll), ok), ok);
    if (!mz && !same) bm = f64_div(phi_min, 1. + f64_div(f64_half(ad, ok), f64_from(f64_bits(phi_min) & 0x7fffffffffffffffll), ok), ok);
    const double q4 = up ? 0.25 : -0.25;
    const double il = fma(q4, ad, sl + qi * d), ir = fma(-q4, ad, sr - qj * d);
    const double al = up ? f64_max(bm, f64_min(il, xl)) : f64_min(bp, f64_max(il, xl));
    const double ar = up ? f64_min(bp, f64_max(ir, xr)) : f64_max(bm, f64_min(ir, xr));
    xl = same ? sl : al;
    xr = same ? sr : ar;
}

// One side of temporal (add_temporal): X the limited spatial state, v the cell's velocity in
// the states' frame; the state reverts to X where density or pressure would turn negative
// (returns true).
PHD_HD __forceinline__ bool half_step64(double *X, const double *p, const double *g, const double *v, double gamma,
                                        double dt, bool &ok) {
    const double y = f64_rcp(p[0], ok), gp = gamma * p[3];
    double x0 = X[0], x1 = X[1] - f64_div_by(dt * g[6], p[0], y, ok), x2 = X[2] - f64_div_by(dt * g[7], p[0], y, ok),
           x3 = X[3];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const double div = g[2 + 3 * k], dv = dt * v[k];
        x0 = x0 - dt * (p[0] * div + v[k] * g[k]);
        x3 = x3 - dt * (gp * div + v[k] * g[6 + k]);
        x1 = x1 - dv * g[2 + k];
        x2 = x2 - dv * g[4 + k];
    }
    if (f64_neg(x0) || f64_neg(x3)) return true;
    X[0] = x0;
    X[1] = x1;
    X[2] = x2;
    X[3] = x3;
    return false;
}

// What a face reads.
struct Face64 {
    double pi[4], pj[4], gi[8], gj[8], w[2];
    double xi[2], xj[2], ci[2], cj[2], com[2];      // generators, centroid offsets, face centroid
};

// The largest magnitude of a face's inputs for which no step can leave the doubles' range
// (states below 2^240 after the half step, energy fluxes below 2^960).
constexpr unsigned F64_FACE_MAX = (1023u + 80u) << 20;

// The states of one face (face_spatial_f64 and temporal, or the cells' own values).
PHD_HD __forceinline__ bool states64(const Face64 &A, const Gas64 &C, double dt_half, bool boost, bool linear, bool gizmo,
                                     double *L, double *R) {
    bool ok = true;
    unsigned big = f64_magmax(f64_magmax(f64_magmax(0u, dt_half), A.w[0]), A.w[1]);
#pragma unroll
    for (int f = 0; f < 4; f++) {
        big = f64_magmax(f64_magmax(big, A.pi[f]), A.pj[f]);
        L[f] = A.pi[f];
        R[f] = A.pj[f];
    }
    if (boost) {
#pragma unroll
        for (int k = 0; k < 2; k++) { L[1 + k] = A.pi[1 + k] - A.w[k]; R[1 + k] = A.pj[1 + k] - A.w[k]; }
    }
    if (linear) {
        double sl[4], sr[4], si[2], sj[2], dx[2];
#pragma unroll
        for (int r = 0; r < 8; r++) big = f64_magmax(f64_magmax(big, A.gi[r]), A.gj[r]);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            si[k] = A.com[k] - (A.xi[k] + A.ci[k]);
            sj[k] = A.com[k] - (A.xj[k] + A.cj[k]);
            dx[k] = A.xj[k] - A.xi[k];
            big = f64_magmax(f64_magmax(big, si[k]), sj[k]);
        }
#pragma unroll
        for (int f = 0; f < 4; f++) {
            sl[f] = L[f];
            sr[f] = R[f];
            L[f] = (L[f] + A.gi[2 * f] * si[0]) + A.gi[2 * f + 1] * si[1];
            R[f] = (R[f] + A.gj[2 * f] * sj[0]) + A.gj[2 * f + 1] * sj[1];
        }
        if (gizmo) {
            const double mi = f64_sqrt(si[0] * si[0] + si[1] * si[1], ok), mj = f64_sqrt(sj[0] * sj[0] + sj[1] * sj[1], ok);
            const double md = f64_sqrt(dx[0] * dx[0] + dx[1] * dx[1], ok), y = f64_rcp(md, ok);
            const double qi = f64_div_by(mi, md, y, ok), qj = f64_div_by(mj, md, y, ok);
#pragma unroll
            for (int f = 0; f < 4; f++) gizmo64(sl[f], sr[f], A.pi[f], A.pj[f], qi, qj, L[f], R[f], ok);
            if (f64_neg(L[0]) || f64_neg(L[3])) {
#pragma unroll
                for (int f = 0; f < 4; f++) L[f] = sl[f];
            }
            if (f64_neg(R[0]) || f64_neg(R[3])) {
#pragma unroll
                for (int f = 0; f < 4; f++) R[f] = sr[f];
            }
        }
        half_step64(L, A.pi, A.gi, sl + 1, C.g, dt_half, ok);
        half_step64(R, A.pj, A.gj, sr + 1, C.g, dt_half, ok);
    }
    return ok && big < F64_FACE_MAX && C.ok;
}

}  // namespace phd
