// phd_exact64.cuh -- the exact Riemann flux of the FP64 path in few FP64 instructions.
//
// ex_get_pstar and exact_flux<double> (phd_physics.cuh) statement by statement -- the same guess,
// Newton iteration, convergence test and sampling -- with the quotients and roots of
// phd_fp64.cuh (IEEE results) and its fixed-point powers, which are rounded to within 0.51 units
// of the last place where the library's are within 2.  A pressure function and its derivative
// take one logarithm between them, the powers at p* serve the sampled state too, and the
// right side is sampled as the mirrored left one.  Twenty library powers a warp made up most of
// the 2263 FP64 instructions of the face kernel; 340 are left, and 962 -> 209 us at 197,000
// faces (point explosion).  A face outside the helpers' windows (vacuum,
// non-finite states) returns false and takes the plain path.
#pragma once
#include "phd_face64.cuh"

namespace phd {

struct Exact64 {
    double g, gm1, gp1, y_gm1, y_gp1, z, e2, inv_z, inv_g, two_gp1, half_gm1, gm1_gp1, gm1_2g, e_d, e_p;
};

inline Exact64 exact64(double gamma) {
    Exact64 X;
    X.g = gamma;
    X.gm1 = gamma - 1.;
    X.gp1 = gamma + 1.;
    X.y_gm1 = 1. / X.gm1;
    X.y_gp1 = 1. / X.gp1;
    X.z = X.gm1 / (2. * gamma);
    X.e2 = (-X.gp1) / (2. * gamma);
    X.inv_z = (2. * gamma) / X.gm1;
    X.inv_g = 1. / gamma;
    X.two_gp1 = 2. / X.gp1;
    X.half_gm1 = 0.5 * X.gm1;
    X.gm1_gp1 = X.gm1 / X.gp1;
    X.gm1_2g = X.gm1 / (2. * gamma);
    X.e_d = 2. / X.gm1;
    X.e_p = (2. * gamma) / X.gm1;
    return X;
}

// The two halves of a power out of line: with nine of them inlined, waiting for instructions
// made up a quarter of the stalls (step of 256 x 256 cells 349 -> 312 us).
#ifdef __CUDACC__
#define PHD_CALL __host__ __device__ __noinline__ inline
#else
#define PHD_CALL inline
#endif
PHD_CALL Log64 log2_call(double x) { return log2_fix(x); }
PHD_CALL double exp2_call(const Log64 &l, double y, bool &ok) { return exp2_fix(l, y, ok); }

PHD_HD __forceinline__ double pow_fix(double x, double y, bool &ok) {
    ok = ok && log2_ok(x);
    return exp2_call(log2_call(x), y, ok);
}

// One side of the pressure function.
struct Side64 {
    double d, p, c, yp, k, cd, ycd;        // reciprocal seeds of p and c d; 2 c / (g - 1)
    double A, B;                           // 2 / ((g + 1) d), (g - 1) / (g + 1) p
};

PHD_HD __forceinline__ Side64 side64(double d, double p, double c, const Exact64 &X, bool &ok) {
    Side64 S;
    S.d = d;
    S.p = p;
    S.c = c;
    S.yp = f64_rcp(p, ok);
    S.k = f64_div_by(2. * c, X.gm1, X.y_gm1, ok);
    S.cd = c * d;
    S.ycd = f64_rcp(S.cd, ok);
    S.A = f64_div(2., S.d * X.gp1, ok);
    S.B = f64_div_by(S.p * X.gm1, X.gp1, X.y_gp1, ok);
    return S;
}

// ex_p_func and, with deriv, ex_p_func_deriv at p_old; q and its logarithm go back from a
// rarefaction side (the power (p_old/p)^z in pz).
PHD_HD __forceinline__ void p_func64(const Side64 &S, const Exact64 &X, double p_old, bool deriv, double &f, double &df,
                                     double &pz, Log64 &l, bool &ok) {
    if (f64_le(p_old, S.p)) {
        const double q = f64_div_by(p_old, S.p, S.yp, ok);
        ok = ok && log2_ok(q);
        l = log2_call(q);
        pz = exp2_call(l, X.z, ok);
        f = S.k * (pz - 1.);
        if (deriv) df = f64_div_by(exp2_call(l, X.e2, ok), S.cd, S.ycd, ok);
    } else {
        const double e = p_old + S.B, y = f64_rcp(e, ok);
        const double s = f64_sqrt(f64_div_by(S.A, e, y, ok), ok), dp = p_old - S.p;
        f = dp * s;
        if (deriv) df = s * fma(-0.5, f64_div_by(dp, e, y, ok), 1.);
    }
}

// ex_p_guess.
PHD_HD __forceinline__ double p_guess64(const Side64 &L, double ul, const Side64 &R, double ur, const Exact64 &X,
                                        bool &ok) {
    const double du = ur - ul;
    const double ppv = f64_half(fma(-0.25, (du * (L.d + R.d)) * (L.c + R.c), L.p + R.p), ok);
    const long long kl = f64_key(L.p), kr = f64_key(R.p), kv = f64_key(ppv);
    const long long kmin = kl < kr ? kl : kr, kmax = kl < kr ? kr : kl, k2 = kmin + (1ll << 52);
    // p_max / p_min <= 2: one unit above 2 p_min may still round to 2
    bool near2 = kmax <= k2;
    if (kmax == k2 + 1) near2 = f64_le(f64_div(f64_from(kmax), f64_from(kmin), ok), 2.);
    if (near2 && kmin <= kv && kv <= kmax) return ppv;
    if (kv <= kmin) {
        const double ycl = f64_rcp(L.c, ok), ycr = f64_rcp(R.c, ok);
        const double plr = pow_fix(f64_div_by(L.p, R.p, R.yp, ok), X.z, ok);
        double us = (f64_div_by(plr * ul, L.c, ycl, ok) + f64_div_by(ur, R.c, ycr, ok)) +
                    f64_div_by(2. * (plr - 1.), X.gm1, X.y_gm1, ok);
        us = f64_div(us, f64_div_by(plr, L.c, ycl, ok) + f64_div_by(1., R.c, ycr, ok), ok);
        const double bl = 1. + f64_div(X.gm1 * (ul - us), 2. * L.c, ok), br = 1. + f64_div(X.gm1 * (us - ur), 2. * R.c, ok);
        return .5 * (L.p * pow_fix(bl, X.inv_z, ok) + R.p * pow_fix(br, X.inv_z, ok));
    }
    const double gl = f64_sqrt(f64_div(L.A, L.B + ppv, ok), ok), gr = f64_sqrt(f64_div(R.A, R.B + ppv, ok), ok);
    return f64_div((gl * L.p + gr * R.p) - du, gr + gl, ok);
}

PHD_HD __forceinline__ bool exact64_flux(const double *L, const double *R, const double *n, const double *w,
                                         const Exact64 &X, int max_iter, double *f, bool *failed) {
    bool ok = f64_pos(L[3]) && f64_pos(R[3]) && f64_pos(L[0]) && f64_pos(R[0]);
    const double ul = L[1] * n[0] + L[2] * n[1], ur = R[1] * n[0] + R[2] * n[1];
    const Side64 A = side64(L[0], L[3], f64_sqrt(f64_div(X.g * L[3], L[0], ok), ok), X, ok);
    const Side64 B = side64(R[0], R[3], f64_sqrt(f64_div(X.g * R[3], R[0], ok), ok), X, ok);
    if (!ok) return false;
    // p* (ex_get_pstar)
    const double TOL = 1.0e-6;
    double p_old = p_guess64(A, ul, B, ur, X, ok), fl = 0., fr = 0., pzl = 1., pzr = 1.;
    Log64 ll = {0, false, 0ull}, lr = ll;
    // one round more than there are Newton steps: the last one forms the functions at p*
    bool conv = false, last = max_iter <= 0;
    for (int it = 1; ok; it++) {
        double dl = 0., dr = 0.;
        p_func64(A, X, p_old, !last, fl, dl, pzl, ll, ok);
        p_func64(B, X, p_old, !last, fr, dr, pzr, lr, ok);
        if (last) break;
        double p_new = p_old - f64_div(((fl + fr) + ur) - ul, dl + dr, ok);
        const double t = f64_div(p_new - p_old, p_new + p_old, ok);
        conv = f64_le(2. * f64_from(f64_bits(t) & 0x7fffffffffffffffll), TOL);
        if (!conv && f64_neg(p_new)) p_new = TOL;
        p_old = p_new;
        last = conv || it >= max_iter;
    }
    if (!ok) return false;
    const double p_new = p_old;
    const double us0 = .5 * (((ul + ur) + fr) - fl);
    // the sampled side, the right one mirrored
    const bool left = f64_le(0., us0);
    const long long sg = left ? 0ll : (long long)0x8000000000000000ull;
    const double d = left ? A.d : B.d, p = left ? A.p : B.p, c = left ? A.c : B.c, yp = left ? A.yp : B.yp;
    const double u = f64_from(f64_bits(left ? ul : ur) ^ sg), us = f64_from(f64_bits(us0) ^ sg);
    double ds = d, ps = p, shift = 0.;
    if (left ? f64_le(p_new, p) : f64_lt(p_new, p)) {
        if (!f64_le(0., u - c)) {
            const double cs = c * (left ? pzl : pzr);
            if (f64_le(us - cs, 0.)) {
                ds = d * exp2_call(left ? ll : lr, X.inv_g, ok);
                ps = p_new;
                shift = us - u;
            } else {
                const double cf = X.two_gp1 * (c + X.half_gm1 * u), r = f64_div(cf, c, ok);
                ok = ok && log2_ok(r);
                const Log64 l = log2_call(r);
                ds = d * exp2_call(l, X.e_d, ok);
                ps = p * exp2_call(l, X.e_p, ok);
                shift = cf - u;
            }
        }
    } else {
        const double r = f64_div(X.gp1 * p_new, (2. * X.g) * p, ok);
        if (!f64_le(0., u - c * f64_sqrt(r + X.gm1_2g, ok))) {
            ds = f64_div(d * (f64_div_by(p_new, p, yp, ok) + X.gm1_gp1),
                         f64_div(p_new * X.gm1, X.gp1 * p, ok) + 1., ok);
            ps = p_new;
            shift = us - u;
        }
    }
    shift = f64_from(f64_bits(shift) ^ sg);
    const double *S = left ? L : R;
    const double v0 = S[1] + shift * n[0], v1 = S[2] + shift * n[1];
    const double vn = v0 * n[0] + v1 * n[1];
    const double e = fma(0.5, ds * (v0 * v0 + v1 * v1), f64_div_by(X.g * ps, X.gm1, X.y_gm1, ok));
    f[0] = ds * vn;
    f[3] = e * vn;
    f[1] = (ds * v0) * vn + ps * n[0];
    f[2] = (ds * v1) * vn + ps * n[1];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const double wf = w[k] * f[0];
        f[3] = f[3] + w[k] * fma(0.5, wf, f[1 + k]);
        f[1 + k] = f[1 + k] + wf;
    }
    if (!conv) *failed = true;
    return ok;
}

}  // namespace phd
