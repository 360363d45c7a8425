// phd_adjface64.cuh -- reverse of one face of the FP64 step (HLL / HLLC) in few FP64 instructions.
//
// The forward is states64 / waves64 (phd_face64.cuh), bit for bit, with the decisions it takes
// kept; the reverse is that of phd_adjoint.cuh (spatial stage with GIZMO, half step, wave
// speeds, star or HLL state, deboost) with the same branches held fixed, arranged for the
// FP64 pipe (phd_fp64.cuh): fused multiply-adds, correctly rounded reciprocals formed by FP32 and
// integer instructions, no forward value recomputed, and no pressure estimate at all where
// both waves are rarefactions (the flux does not depend on it).  What the lean forward
// declines, and a two-rarefaction estimate that does enter the wave speeds, returns false:
// the plain reverse then does the face.
#pragma once
#include "phd_face64.cuh"

namespace phd {

// Decisions of the spatial stage and the half step of one face.
struct StateDecisions {
    unsigned flat, inner_l, outer_l, inner_r, outer_r;          // a bit per field
    bool spat_l, spat_r, half_l, half_r;                        // the states reverted there
    double qi, qj, si[2], sj[2];
};

PHD_HD __forceinline__ double f64_abs(double a) { return f64_from(f64_bits(a) & 0x7fffffffffffffffll); }
PHD_HD __forceinline__ bool opposite64(double a, double b) {
    return (f64_bits(a) ^ f64_bits(b)) < 0 && !f64_zero(a) && !f64_zero(b);
}

// gizmo64 with its decisions.
PHD_HD __forceinline__ void gizmo64_decide(int f, double sl, double sr, double ci, double cj, double &xl, double &xr,
                                           StateDecisions &D, bool &ok) {
    const long long ki = f64_key(ci), kj = f64_key(cj);
    if (ki == kj) {
        D.flat |= 1u << f;
        xl = sl;
        xr = sr;
        return;
    }
    const bool up = ki < kj;
    const double d = sr - sl, h = up ? 0.5 : -0.5, q4 = up ? 0.25 : -0.25;
    // the ordered cells' states are ordered alike; a tie (or, with two face velocities, any
    // other order) is the plain path's
    ok = ok && (up ? f64_pos(d) : f64_neg(d));
    const double ad = f64_abs(d);
    double ol = fma(-h, ad, sl), orr = fma(h, ad, sr);                  // phi_minus / phi_plus
    // a bound of the other sign than its state: the quotient form
    if (opposite64(ol, sl)) ol = f64_div(sl, 1. + f64_div(f64_half(ad, ok), f64_abs(sl), ok), ok);
    if (opposite64(orr, sr)) orr = f64_div(sr, 1. + f64_div(f64_half(ad, ok), f64_abs(sr), ok), ok);
    const double il = fma(q4, ad, sl + D.qi * d), ir = fma(-q4, ad, sr - D.qj * d);
    const long long kil = f64_key(il), kir = f64_key(ir), kxl = f64_key(xl), kxr = f64_key(xr), kol = f64_key(ol),
                    kor = f64_key(orr);
    const bool nl = up ? kil <= kxl : kil >= kxl, nr = up ? kir >= kxr : kir <= kxr;       // inner before the state
    const long long ml = nl ? kil : kxl, mr = nr ? kir : kxr;
    const bool tl = up ? kol >= ml : kol <= ml, tr = up ? kor <= mr : kor >= mr;           // outer before both
    D.outer_l |= (unsigned)tl << f;
    D.outer_r |= (unsigned)tr << f;
    D.inner_l |= (unsigned)(nl && !tl) << f;
    D.inner_r |= (unsigned)(nr && !tr) << f;
    xl = tl ? ol : (nl ? il : xl);
    xr = tr ? orr : (nr ? ir : xr);
}

PHD_HD __forceinline__ bool states64_decide(const Face64 &A, const Gas64 &C, double dt_half, bool boost, bool gizmo,
                                            double *sl, double *sr, double *L, double *R, StateDecisions &D) {
    bool ok = true;
    unsigned big = f64_magmax(f64_magmax(f64_magmax(0u, dt_half), A.w[0]), A.w[1]);
    double dx[2];
#pragma unroll
    for (int f = 0; f < 4; f++) {
        big = f64_magmax(f64_magmax(big, A.pi[f]), A.pj[f]);
        sl[f] = A.pi[f];
        sr[f] = A.pj[f];
    }
    if (boost) {
#pragma unroll
        for (int k = 0; k < 2; k++) { sl[1 + k] = A.pi[1 + k] - A.w[k]; sr[1 + k] = A.pj[1 + k] - A.w[k]; }
    }
#pragma unroll
    for (int r = 0; r < 8; r++) big = f64_magmax(f64_magmax(big, A.gi[r]), A.gj[r]);
#pragma unroll
    for (int k = 0; k < 2; k++) {
        D.si[k] = A.com[k] - (A.xi[k] + A.ci[k]);
        D.sj[k] = A.com[k] - (A.xj[k] + A.cj[k]);
        dx[k] = A.xj[k] - A.xi[k];
        big = f64_magmax(f64_magmax(big, D.si[k]), D.sj[k]);
    }
#pragma unroll
    for (int f = 0; f < 4; f++) {
        L[f] = (sl[f] + A.gi[2 * f] * D.si[0]) + A.gi[2 * f + 1] * D.si[1];
        R[f] = (sr[f] + A.gj[2 * f] * D.sj[0]) + A.gj[2 * f + 1] * D.sj[1];
    }
    D.flat = D.inner_l = D.outer_l = D.inner_r = D.outer_r = 0u;
    D.spat_l = D.spat_r = false;
    D.qi = D.qj = 0.;
    if (gizmo) {
        const double mi = f64_sqrt(D.si[0] * D.si[0] + D.si[1] * D.si[1], ok);
        const double mj = f64_sqrt(D.sj[0] * D.sj[0] + D.sj[1] * D.sj[1], ok);
        const double md = f64_sqrt(dx[0] * dx[0] + dx[1] * dx[1], ok), y = f64_rcp(md, ok);
        D.qi = f64_div_by(mi, md, y, ok);
        D.qj = f64_div_by(mj, md, y, ok);
#pragma unroll
        for (int f = 0; f < 4; f++) gizmo64_decide(f, sl[f], sr[f], A.pi[f], A.pj[f], L[f], R[f], D, ok);
        D.spat_l = f64_neg(L[0]) || f64_neg(L[3]);
        D.spat_r = f64_neg(R[0]) || f64_neg(R[3]);
#pragma unroll
        for (int f = 0; f < 4; f++) {
            L[f] = D.spat_l ? sl[f] : L[f];
            R[f] = D.spat_r ? sr[f] : R[f];
        }
    }
    D.half_l = half_step64(L, A.pi, A.gi, sl + 1, C.g, dt_half, ok);
    D.half_r = half_step64(R, A.pj, A.gj, sr + 1, C.g, dt_half, ok);
    return ok && big < F64_FACE_MAX && C.ok;
}

// waves64 with what its reverse reads.
struct WaveTape64 {
    double cl, cr, du, ds, cs, gl, gr, iS, idl, idr, ql, qr, ps, iD, bl, br;
    int kind;                      // 0: the linearised pressure, 2: two shocks, 1: no pressure needed
    bool pv_pos, shl, shr;
};

PHD_HD __forceinline__ bool waves64_tape(double dl, double ul, double pl, double dr, double ur, double pr, const Gas64 &C,
                                         WaveTape64 &T, double &sl, double &sc, double &sr, double &ml, double &mr) {
    bool ok = f64_pos(pl) && f64_pos(pr);
    T.cl = f64_sqrt(f64_div(C.g * pl, dl, ok), ok);
    T.cr = f64_sqrt(f64_div(C.g * pr, dr, ok), ok);
    ok = ok && f64_lt(1.0E-10, T.cl) && f64_lt(1.0E-10, T.cr);
    T.cs = T.cl + T.cr;
    T.du = ul - ur;
    T.ds = dl + dr;
    const double pv = f64_half(fma(0.25, (T.du * T.ds) * T.cs, pl + pr), ok);
    T.pv_pos = f64_pos(pv);
    double ps = f64_neg(pv) ? 0. : pv;
    const long long kl = f64_key(pl), kr = f64_key(pr), ks = f64_key(ps);
    const bool lr = kl <= kr;
    const long long kmin = lr ? kl : kr, kmax = lr ? kr : kl;
    T.kind = 0;
    T.gl = T.gr = T.iS = T.idl = T.idr = 0.;
    if (kmax < kmin + (1ll << 52) && kmin < ks && ks < kmax) {
    } else if (ks <= kmin) {
        T.kind = 1;
        const double dp = lr ? pr - pl : pl - pr;
        const bool same = f64_zero(dp) && f64_zero(T.du) && f64_bits(dl) == f64_bits(dr) &&
                          C.half_gm1f * fabsf(f64_to_f32(ul)) < 0.15f * f64_to_f32(T.cl);
        if (!(same || trrs_below(dp, lr ? pr : pl, T.du, lr ? T.cr : T.cl, T.cs, ul, ur, C))) return false;
    } else {
        T.kind = 2;
        const double el = ps + pl * C.gm1_gp1, er = ps + pr * C.gm1_gp1;
        T.gl = f64_sqrt(f64_div(f64_div(2., C.gp1 * dl, ok), el, ok), ok);
        T.gr = f64_sqrt(f64_div(f64_div(2., C.gp1 * dr, ok), er, ok), ok);
        const double S = T.gl + T.gr;
        T.idl = f64_rcp(el, ok);
        T.idr = f64_rcp(er, ok);
        T.iS = f64_rcp(S, ok);
        ps = f64_div_by((T.gl * pl + T.gr * pr) + T.du, S, T.iS, ok);
    }
    T.ps = ps;
    T.shl = T.kind != 1 && !(f64_key(ps) <= kl);
    T.shr = T.kind != 1 && !(f64_key(ps) <= kr);
    T.ql = T.qr = 1.;
    double al = T.cl, ar = T.cr;
    if (T.shl) {
        T.ql = f64_sqrt(1. + C.gp1_2g * (f64_div(ps, pl, ok) - 1.), ok);
        al = T.cl * T.ql;
    }
    if (T.shr) {
        T.qr = f64_sqrt(1. + C.gp1_2g * (f64_div(ps, pr, ok) - 1.), ok);
        ar = T.cr * T.qr;
    }
    sl = ul - al;
    sr = ur + ar;
    T.bl = sl - ul;
    T.br = sr - ur;
    ml = dl * T.bl;
    mr = dr * T.br;
    const double D = ml - mr;
    T.iD = f64_rcp(D, ok);
    sc = f64_div_by(((pr - pl) + (dl * ul) * T.bl) - (dr * ur) * T.br, D, T.iD, ok);
    return ok;
}

// Reverse: adjoints of the speeds and of m = d (s - u) -> of the sides' density, normal
// velocity and pressure (accumulated).
PHD_HD __forceinline__ void waves64_rev(const WaveTape64 &T, double dl, double ul, double pl, double dr, double ur,
                                        double pr, const Gas64 &C, double ml, double mr, double sc, double asl, double asc,
                                        double asr, double aml, double amr, double &adl, double &aul, double &apl,
                                        double &adr, double &aur, double &apr, bool &ok) {
    const double ipl = f64_rcp(pl, ok), ipr = f64_rcp(pr, ok), irl = f64_rcp(dl, ok), irr = f64_rcp(dr, ok);
    // sc = (p_r - p_l + u_l m_l - u_r m_r) / (m_l - m_r)
    const double aN = asc * T.iD;
    apr += aN;
    apl -= aN;
    aul = fma(aN, ml, aul);
    aur = fma(-aN, mr, aur);
    aml = fma(aN, ul - sc, aml);
    amr = fma(-aN, ur - sc, amr);
    adl = fma(aml, T.bl, adl);
    adr = fma(amr, T.br, adr);
    const double abl = aml * dl, abr = amr * dr;
    asl += abl;
    asr += abr;
    // s_l = u_l - c_l q_l, s_r = u_r + c_r q_r
    aul += asl - abl;
    aur += asr - abr;
    double acl = -asl * T.ql, acr = asr * T.qr, aps = 0.;
    if (T.shl) {
        const double t = (-0.5 * C.gp1_2g) * (asl * T.cl) * f64_rcp(T.ql, ok) * ipl;
        aps += t;
        apl = fma(-t * T.ps, ipl, apl);
    }
    if (T.shr) {
        const double t = (0.5 * C.gp1_2g) * (asr * T.cr) * f64_rcp(T.qr, ok) * ipr;
        aps += t;
        apr = fma(-t * T.ps, ipr, apr);
    }
    if (T.kind != 1) {
        double apv = aps;
        if (T.kind == 2) {
            const double a = aps * T.iS;
            const double hl = (0.5 * a) * (pl - T.ps) * T.gl, hr = (0.5 * a) * (pr - T.ps) * T.gr;
            apl = fma(a, T.gl, apl);
            apr = fma(a, T.gr, apr);
            aul += a;
            aur -= a;
            adl = fma(-hl, irl, adl);
            adr = fma(-hr, irr, adr);
            const double tl = hl * T.idl, tr = hr * T.idr;
            apl = fma(-tl, C.gm1_gp1, apl);
            apr = fma(-tr, C.gm1_gp1, apr);
            apv = -(tl + tr);
        }
        if (T.pv_pos) {
            const double h = 0.5 * apv, e = 0.125 * apv, dc = e * T.cs;
            apl += h;
            apr += h;
            const double au = dc * T.ds, ad = dc * T.du, ac = (e * T.du) * T.ds;
            aul += au;
            aur -= au;
            adl += ad;
            adr += ad;
            acl += ac;
            acr += ac;
        }
    }
    // c = sqrt(g p / d)
    const double hl = (0.5 * acl) * T.cl, hr = (0.5 * acr) * T.cr;
    apl = fma(hl, ipl, apl);
    adl = fma(-hl, irl, adl);
    apr = fma(hr, ipr, apr);
    adr = fma(-hr, irr, adr);
}

// Adjoint of hll64: accumulates into aL, aR.
template <bool HLLC>
PHD_HD __forceinline__ bool hll64_adj(const double *L, const double *R, const double *n, const double *w, const Gas64 &C,
                                      bool boost, const double *aFin, double *aL, double *aR) {
    const double dl = L[0], pl = L[3], dr = R[0], pr = R[3];
    const double Vnl = L[1] * n[0] + L[2] * n[1], Vnr = R[1] * n[0] + R[2] * n[1];
    const double wn = boost ? 0. : w[0] * n[0] + w[1] * n[1];
    WaveTape64 T;
    double sl, sc, sr, ml, mr;
    bool ok = waves64_tape(dl, Vnl, pl, dr, Vnr, pr, C, T, sl, sc, sr, ml, mr);
    if (!ok) return false;
    double aF[4] = {aFin[0], aFin[1], aFin[2], aFin[3]};
    if (boost) {
        aF[1] = fma(w[0], aFin[3], aFin[1]);
        aF[2] = fma(w[1], aFin[3], aFin[2]);
        aF[0] = fma(0.5 * fma(w[0], w[0], w[1] * w[1]), aFin[3], fma(w[1], aFin[2], fma(w[0], aFin[1], aFin[0])));
    }
    double asl = 0., asc = 0., asr = 0., aml = 0., amr = 0.;
    double adl = 0., adr = 0., apl = 0., apr = 0., aVl = 0., aVr = 0.;
    const bool data_l = f64_le(wn, sl), data_r = !data_l && !f64_le(wn, sr);
    const double ig = C.y_gm1;
    bool waves = true;
    if (HLLC || data_l || data_r) {
        const bool left = data_l || (!data_r && f64_le(wn, sc));
        const double d = left ? dl : dr, p = left ? pl : pr, Vn = left ? Vnl : Vnr;
        const double v0 = left ? L[1] : R[1], v1 = left ? L[2] : R[2];
        const double vsq = fma(v0, v0, v1 * v1), e = fma(0.5 * d, vsq, p * ig);
        const double fv = fma(aF[1], v0, aF[2] * v1), fn = fma(aF[1], n[0], aF[2] * n[1]);
        double ad, ap, aV, ae, av0, av1;
        if (data_l || data_r) {
            const double u = Vn - wn, t = fma(d, fv, fma(aF[0], d, aF[3] * e));      // adjoint of u
            ad = fma(u, fv, aF[0] * u);
            ap = fma(aF[3], Vn, fn);
            aV = fma(aF[3], p, t);
            ae = aF[3] * u;
            const double du = d * u;
            av0 = aF[1] * du;
            av1 = aF[2] * du;
            waves = false;
        } else {
            const double s = left ? sl : sr, m = left ? ml : mr;
            const double sw = s - wn, ib = f64_rcp(s - sc, ok), id = f64_rcp(d, ok), im = f64_rcp(m, ok);
            const double f1 = m * ib, f1w = f1 * sw, q = sc - Vn, frho = f1w - m, t = p * im, st = sc + t;
            const double ed = e * id, Q = fma(q, st, ed);
            const double afr = aF[0] + fv;
            av0 = aF[1] * frho;
            av1 = aF[2] * frho;
            const double aQ = aF[3] * f1w;
            ae = fma(aQ, id, aF[3] * (Vn - s));
            ad = -aQ * ed * id;
            const double aq = fma(aQ, st, fn * f1w);
            const double at = aQ * q;
            const double af1w = fma(fn, q, fma(aF[3], Q, afr));
            double am = fma(-at * t, im, -afr);
            ap = fma(at, im, fma(aF[3], Vn, fn));
            aV = fma(aF[3], e + p, -aq);
            const double a1 = af1w * sw, ab = -a1 * f1 * ib;
            am = fma(a1, ib, am);
            const double as = fma(af1w, f1, fma(-aF[3], e, ab));
            asc = (at + aq) - ab;
            aml = left ? am : 0.;
            amr = left ? 0. : am;
            asl = left ? as : 0.;
            asr = left ? 0. : as;
        }
        ad = fma(0.5 * vsq, ae, ad);
        ap = fma(ig, ae, ap);
        const double a2 = d * ae;                      // 2 (d/2) ae, the adjoint of v^2 times 2
        av0 = fma(a2, v0, av0);
        av1 = fma(a2, v1, av1);
        if (left) {
            adl = ad;
            apl = ap;
            aVl = aV;
            aL[1] += av0;
            aL[2] += av1;
        } else {
            adr = ad;
            apr = ap;
            aVr = aV;
            aR[1] += av0;
            aR[2] += av1;
        }
    } else {
        // f = (fac1 (F_l - s_l U_l) - fac2 (F_r - s_r U_r)) / fac3
        const double fac1 = sr - wn, fac2 = sl - wn, i3 = f64_rcp(sr - sl, ok);
        double af3 = 0., g[2];
#pragma unroll
        for (int s = 0; s < 2; s++) {
            const double *S = s ? R : L;
            const double d = S[0], p = S[3], Vn = s ? Vnr : Vnl, k = s ? sr : sl, fac = s ? -fac2 : fac1;
            const double vsq = fma(S[1], S[1], S[2] * S[2]), e = fma(0.5 * d, vsq, p * ig);
            const double fv = fma(aF[1], S[1], aF[2] * S[2]), fn = fma(aF[1], n[0], aF[2] * n[1]);
            const double r = Vn - k, du = fma(fv, d, fma(aF[0], d, aF[3] * e));      // sum_c a_c U_c
            // G = sum_c a_c (F_c - k U_c) = du r + fn p + aF3 p Vn
            g[s] = i3 * fma(du, r, p * fma(aF[3], Vn, fn));
            af3 = fma(-g[s] * i3, fac, af3);
            const double z = fac * i3, ae = z * aF[3] * r;
            const double ad = fma(0.5 * vsq, ae, z * r * (aF[0] + fv));
            const double ap = fma(ig, ae, z * fma(aF[3], Vn, fn));
            const double aV = z * fma(aF[3], p, du);
            const double zr = z * r * d, a2 = d * ae;
            double *aS = s ? aR : aL;
            aS[1] += fma(aF[1], zr, a2 * S[1]);
            aS[2] += fma(aF[2], zr, a2 * S[2]);
            if (s) { adr = ad; apr = ap; aVr = aV; asr = -z * du; }
            else { adl = ad; apl = ap; aVl = aV; asl = -z * du; }
        }
        asr += g[0] + af3;                             // fac1 = s_r - w.n, fac3 = s_r - s_l
        asl -= g[1] + af3;                             // fac2 = s_l - w.n
    }
    if (waves)
        waves64_rev(T, dl, Vnl, pl, dr, Vnr, pr, C, ml, mr, sc, asl, asc, asr, aml, amr, adl, aVl, apl, adr, aVr, apr, ok);
    aL[0] += adl;
    aL[3] += apl;
    aR[0] += adr;
    aR[3] += apr;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        aL[1 + k] = fma(aVl, n[k], aL[1 + k]);
        aR[1 + k] = fma(aVr, n[k], aR[1 + k]);
    }
    return ok;
}

// Reverse of one side's half step and spatial stage: a the adjoint of the side's state, X
// selecting the left (0) or right (1) side; as, ao receive the adjoints of the side's own and
// of the other cell's state, ap (rho, -, -, p) and av (velocity in the states' frame) the half
// step's, ag the gradient's.
PHD_HD __forceinline__ void side64_rev(const double *a, bool half_rev, bool spat_rev, bool gizmo, bool right,
                                       const StateDecisions &D, const double *p, const double *g, const double *so,
                                       const double *oo,
                                       double gamma, double dt, double *as, double *ao, double *ag, double &arho,
                                       double &aprs, bool &ok) {
    const double *sep = right ? D.sj : D.si, *v = so + 1;
    double a1 = a[1], a2 = a[2], av0 = 0., av1 = 0.;
    arho = aprs = 0.;
#pragma unroll
    for (int r = 0; r < 8; r++) ag[r] = 0.;
    if (!half_rev) {
        const double y = f64_rcp(p[0], ok);
        const double b0 = -dt * a[0], b1 = -dt * a1, b2 = -dt * a2, b3 = -dt * a[3];
        const double gp = gamma * p[3], div = g[2] + g[5], t = fma(p[0], b0, gp * b3);
        ag[0] = v[0] * b0;
        ag[1] = v[1] * b0;
        ag[2] = fma(v[0], b1, t);
        ag[3] = v[1] * b1;
        ag[4] = v[0] * b2;
        ag[5] = fma(v[1], b2, t);
        ag[6] = fma(v[0], b3, b1 * y);
        ag[7] = fma(v[1], b3, b2 * y);
        arho = fma(div, b0, -(y * y) * fma(g[6], b1, g[7] * b2));
        aprs = gamma * div * b3;
        av0 = fma(g[0], b0, fma(g[2], b1, fma(g[4], b2, g[6] * b3)));
        av1 = fma(g[1], b0, fma(g[3], b1, fma(g[5], b2, g[7] * b3)));
    }
    const double q = right ? D.qj : D.qi;
    const unsigned inner = right ? D.inner_r : D.inner_l, outer = right ? D.outer_r : D.outer_l;
#pragma unroll
    for (int f = 0; f < 4; f++) {
        const double af = a[f];
        double x = af, s = 0., o = 0.;                 // through the slope; own and other state's shares
        if (spat_rev) {
            x = 0.;
            s = af;
        } else if (gizmo) {
            const unsigned b = 1u << f;
            if (D.flat & b) {
                x = 0.;
                s = af;
            } else if (outer & b) {
                // s - (other - s)/2 or, where that would change sign, s / k with
                // k = 1 + |other - s| / (2 |s|)
                const double h = 0.5 * (oo[f] - so[f]);
                x = 0.;
                s = 1.5 * af;
                o = -0.5 * af;
                if (opposite64(so[f] - h, so[f])) {
                    const double ab = f64_abs(so[f]), y = ab * f64_rcp(ab + f64_abs(h), ok), t = af * y;
                    o = -0.5 * t * y;
                    s = fma(2., t, o);
                }
            } else if (inner & b) {                    // s + (q + 1/4) (other - s)
                x = 0.;
                o = fma(q, af, 0.25 * af);
                s = af - o;
            }
        }
        as[f] = x + s;
        ao[f] = o;
        ag[2 * f] = fma(x, sep[0], ag[2 * f]);
        ag[2 * f + 1] = fma(x, sep[1], ag[2 * f + 1]);
    }
    as[1] += av0;
    as[2] += av1;
}

}  // namespace phd
