// phd_adj.cu -- hand-written adjoint of one FP64 step (mesh, face velocities, dt fixed).
//
// Forward step (real-cell conserved totals U -> U'):
//   ghost refresh -> primitives -> limited gradients -> face states (spatial +
//   GIZMO + MUSCL-Hancock half step) -> HLL/HLLC flux + deboost -> segmented update.
// Reverse, three deterministic kernels (no atomics; every sum is a per-thread loop):
//   k_adj_face     per face: flux adjoint dt*A*(lam'_j - lam'_i) through Riemann,
//                  temporal and spatial stages -> 24 per-face adjoint values
//   k_adj_cell     per cell: sum its faces' contributions; a real cell with its ghost rows
//                  folded in, through the reverse of the limited gradient -> per-entry
//                  neighbour adjoints and the cell's own adjoint (k_adj_cell_taped after a taped
//                  forward step, four threads a cell)
//   k_adj_final    per real cell: own and ghost rows' sums and the neighbours' parts through
//                  the reverse of the primitive recovery, lam = lam' + J^T lam_prim

#include "phd_common.cuh"
#include "phd_physics.cuh"
#include "phd_adjoint.cuh"
#include "phd_ref.cuh"
#include "phd_adjface64.cuh"

namespace phd {

constexpr int BA = 256;
constexpr int FACE_ADJ = 24;   // api[4] apj[4] agi[8] agj[8]

// add_spatial (reference geometry) for one face, split into a forward pass that keeps
// what the reverse needs (the "tape") and the reverse itself, so the adjoint kernel
// evaluates the forward once.  The forward is face_spatial_f64's arithmetic in the
// same order (so the same branches): boosted cell states, extrapolation along the
// centroid separations, GIZMO pair limiter, revert where density or pressure < 0.
struct SpatialTape {
    double sl[4], sr[4], L0[4], R0[4], sepi[2], sepj[2], sepi_mag, sepj_mag, diff_mag;
    bool revL, revR;
};

__device__ __forceinline__ void spatial_fwd_f64(const phd_mesh &M, int m, int i, int j, const double *pi,
                                                const double *pj, const double *gi, const double *gj,
                                                const double *w, bool boost, bool gizmo, SpatialTape &t,
                                                double *Ls, double *Rs) {
    const int n = M.n_cells, F = M.n_faces;
    for (int f = 0; f < 4; f++) { t.sl[f] = pi[f]; t.sr[f] = pj[f]; }
    if (boost)
        for (int k = 0; k < 2; k++) { t.sl[1 + k] = pi[1 + k] - w[k]; t.sr[1 + k] = pj[1 + k] - w[k]; }
    for (int f = 0; f < 4; f++) { t.L0[f] = t.sl[f]; t.R0[f] = t.sr[f]; }
    double diff_mag = 0.0, sepi_mag = 0.0, sepj_mag = 0.0;
    for (int k = 0; k < 2; k++) {
        const double fc = M.com[(size_t)k * F + m];
        const double xik = M.x[(size_t)k * n + i], xjk = M.x[(size_t)k * n + j];
        t.sepi[k] = fc - (xik + M.dcom[(size_t)k * n + i]);
        t.sepj[k] = fc - (xjk + M.dcom[(size_t)k * n + j]);
        sepi_mag = sepi_mag + t.sepi[k] * t.sepi[k];
        sepj_mag = sepj_mag + t.sepj[k] * t.sepj[k];
        diff_mag = diff_mag + t_sq(xjk - xik);
        for (int f = 0; f < 4; f++) {
            t.L0[f] = t.L0[f] + gi[f * 2 + k] * t.sepi[k];
            t.R0[f] = t.R0[f] + gj[f * 2 + k] * t.sepj[k];
        }
    }
    t.sepi_mag = sqrt(sepi_mag);
    t.sepj_mag = sqrt(sepj_mag);
    t.diff_mag = sqrt(diff_mag);
    t.revL = t.revR = false;
    for (int f = 0; f < 4; f++) { Ls[f] = t.L0[f]; Rs[f] = t.R0[f]; }
    if (gizmo) {
        for (int f = 0; f < 4; f++)
            gizmo_pair<double>(t.sl[f], t.sr[f], pi[f], pj[f], t.sepi_mag, t.sepj_mag, t.diff_mag, Ls[f], Rs[f]);
        t.revL = (Ls[0] < 0.0 || Ls[3] < 0.0);
        t.revR = (Rs[0] < 0.0 || Rs[3] < 0.0);
        for (int f = 0; f < 4; f++) {
            if (t.revL) Ls[f] = t.sl[f];
            if (t.revR) Rs[f] = t.sr[f];
        }
    }
}

__device__ __forceinline__ void spatial_rev_f64(const SpatialTape &t, const double *pi, const double *pj,
                                                bool gizmo, const double *aL, const double *aR, double *api,
                                                double *apj, double *agi, double *agj) {
    double asl[4] = {0, 0, 0, 0}, asr[4] = {0, 0, 0, 0}, aL0[4] = {0, 0, 0, 0}, aR0[4] = {0, 0, 0, 0};
    if (gizmo) {
        double aL1[4], aR1[4];
        for (int f = 0; f < 4; f++) {
            aL1[f] = t.revL ? 0.0 : aL[f];
            aR1[f] = t.revR ? 0.0 : aR[f];
            if (t.revL) asl[f] += aL[f];
            if (t.revR) asr[f] += aR[f];
        }
        const double si = t.sepi_mag / t.diff_mag, sj = t.sepj_mag / t.diff_mag;
        for (int f = 0; f < 4; f++)
            gizmo_pair_adj_q<double>(t.sl[f], t.sr[f], pi[f], pj[f], si, sj, t.L0[f], t.R0[f], aL1[f], aR1[f],
                                     asl[f], asr[f], aL0[f], aR0[f]);
    } else {
        for (int f = 0; f < 4; f++) { aL0[f] = aL[f]; aR0[f] = aR[f]; }
    }
    for (int f = 0; f < 4; f++) {
        asl[f] += aL0[f];
        asr[f] += aR0[f];
        for (int k = 0; k < 2; k++) {
            agi[f * 2 + k] += aL0[f] * t.sepi[k];
            agj[f * 2 + k] += aR0[f] * t.sepj[k];
        }
        api[f] += asl[f];
        apj[f] += asr[f];
    }
}

// One face on the plain path: 24 values to out.  EXACT: the exact solver's reverse
// (exact_flux_adj); otherwise HLL / HLLC.
template <bool EXACT>
__device__ __forceinline__ void adj_face_body(const phd_mesh &M, const phd_params &P, double dt, const double *prim,
                                              const double *grad, const double *face_w, const double *lam_next, int m,
                                              int i, int j, double *out) {
    const int n = M.n_cells, F = M.n_faces;
    double res[FACE_ADJ];
    for (int q = 0; q < FACE_ADJ; q++) res[q] = 0.0;
    const bool boost = (P.boost != 0);
    const bool linear = P.reconstruction == PHD_LINEAR;
    double pi[4], pj[4], gi[8], gj[8], w[2], nrm[2];
    for (int f = 0; f < 4; f++) { pi[f] = prim[(size_t)f * n + i]; pj[f] = prim[(size_t)f * n + j]; }
    for (int r = 0; r < 8; r++) {
        gi[r] = linear ? grad[(size_t)r * n + i] : 0.0;
        gj[r] = linear ? grad[(size_t)r * n + j] : 0.0;
    }
    for (int k = 0; k < 2; k++) {
        w[k] = face_w ? face_w[(size_t)k * F + m] : 0.0;
        nrm[k] = M.normal[(size_t)k * F + m];
    }
    // flux adjoint from the update U_i -= dt a F, U_j += dt a F (j real)
    const double da = dt * M.area[m];
    const bool jr = M.tag[j] == PHD_REAL_TAG;
    double aF[4];
    for (int q = 0; q < 4; q++)
        aF[q] = da * ((jr ? lam_next[(size_t)q * n + j] : 0.0) - lam_next[(size_t)q * n + i]);
    // forward states (the spatial stage once, its tape kept for the reverse)
    double Ls[4], Rs[4], L[4], R[4];
    SpatialTape tape;
    if (linear) {
        spatial_fwd_f64(M, m, i, j, pi, pj, gi, gj, w, boost, P.gizmo != 0, tape, Ls, Rs);
        for (int f = 0; f < 4; f++) { L[f] = Ls[f]; R[f] = Rs[f]; }
        temporal<double, 2>(L, R, pi, pj, gi, gj, w, P.gamma, 0.5 * dt, boost);
    } else {
        for (int f = 0; f < 4; f++) { L[f] = pi[f]; R[f] = pj[f]; }
        if (boost) for (int k = 0; k < 2; k++) { L[1 + k] -= w[k]; R[1 + k] -= w[k]; }
    }
    double aL[4] = {0, 0, 0, 0}, aR[4] = {0, 0, 0, 0};
    if (EXACT) exact_flux_adj(L, R, nrm, w, P.gamma, P.exact_max_iter, aF, aL, aR);
    else hll_family_adj<double>(P.solver == PHD_HLLC, L, R, nrm, w, P.gamma, boost, aF, aL, aR);
    double *api = res, *apj = res + 4, *agi = res + 8, *agj = res + 16;
    if (linear) {
        double aLs[4] = {0, 0, 0, 0}, aRs[4] = {0, 0, 0, 0};
        temporal_adj<double>(Ls, Rs, pi, pj, gi, gj, w, P.gamma, 0.5 * dt, boost, aL, aR, aLs, aRs, api, apj,
                             agi, agj);
        spatial_rev_f64(tape, pi, pj, P.gizmo != 0, aLs, aRs, api, apj, agi, agj);
    } else {
        for (int f = 0; f < 4; f++) { api[f] += aL[f]; apj[f] += aR[f]; }
    }
    for (int q = 0; q < FACE_ADJ; q++) out[(size_t)q * F + m] = res[q];
}

__device__ __noinline__ void adj_face_plain(const phd_mesh *M, const phd_params *P, double dt, const double *prim,
                                            const double *grad, const double *face_w, const double *lam_next, int m,
                                            int i, int j, double *out) {
    adj_face_body<false>(*M, *P, dt, prim, grad, face_w, lam_next, m, i, j, out);
}

// The exact solver's faces (220 registers).
__global__ void __launch_bounds__(BA) k_adj_face_exact(phd_mesh M, phd_params P, double dt, const double *__restrict__ prim,
                                                       const double *__restrict__ grad,
                                                       const double *__restrict__ face_w,
                                                       const double *__restrict__ lam_next, double *__restrict__ out) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M.n_faces) return;
    const int i = M.pair_i[m], j = M.pair_j[m];
    if (i < 0 || i >= M.n_cells || j < 0 || j >= M.n_cells) {
        for (int q = 0; q < FACE_ADJ; q++) out[(size_t)q * M.n_faces + m] = 0.0;
        return;
    }
    adj_face_body<true>(M, P, dt, prim, grad, face_w, lam_next, m, i, j, out);
}

// HLL / HLLC: the lean reverse (phd_adjface64.cuh), the plain one for the faces it declines.
// Bound by the FP64 pipe; held to 168 registers for 12 warps an SM (the pipe waits on 8 at 255:
// 14.0 against 15.1 ms for 40 steps forward and backward at 128 x 128).  Measured there (50,000
// faces, HLLC, cold caches): 317 -> 67 us, 2157 -> 567 FP64 instructions per warp.
template <bool HLLC>
__global__ void __launch_bounds__(128, 3) k_adj_face(const __grid_constant__ phd_mesh M, const __grid_constant__ phd_params P,
                                                  const __grid_constant__ Gas64 C, double dt,
                                                  const double *__restrict__ prim, const double *__restrict__ grad,
                                                  const double *__restrict__ face_w,
                                                  const double *__restrict__ lam_next, double *__restrict__ out) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M.n_faces) return;
    const int n = M.n_cells, F = M.n_faces;
    const int i = M.pair_i[m], j = M.pair_j[m];
    if (i < 0 || i >= n || j < 0 || j >= n) {
        for (int q = 0; q < FACE_ADJ; q++) out[(size_t)q * F + m] = 0.0;
        return;
    }
    const bool boost = P.boost != 0, linear = P.reconstruction == PHD_LINEAR, gizmo = P.gizmo != 0;
    Face64 A;
#pragma unroll
    for (int f = 0; f < 4; f++) { A.pi[f] = prim[(size_t)f * n + i]; A.pj[f] = prim[(size_t)f * n + j]; }
#pragma unroll
    for (int r = 0; r < 8; r++) {
        A.gi[r] = linear ? grad[(size_t)r * n + i] : 0.0;
        A.gj[r] = linear ? grad[(size_t)r * n + j] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < 2; k++) {
        A.w[k] = face_w ? face_w[(size_t)k * F + m] : 0.0;
        A.xi[k] = M.x[(size_t)k * n + i];
        A.xj[k] = M.x[(size_t)k * n + j];
        A.ci[k] = M.dcom[(size_t)k * n + i];
        A.cj[k] = M.dcom[(size_t)k * n + j];
        A.com[k] = M.com[(size_t)k * F + m];
    }
    const double nrm[2] = {M.normal[m], M.normal[(size_t)F + m]};
    // flux adjoint from the update U_i -= dt a F, U_j += dt a F (j real)
    const double da = dt * M.area[m];
    const bool jr = M.tag[j] == PHD_REAL_TAG;
    double aF[4], sl[4], sr[4], L[4], R[4], aL[4] = {0., 0., 0., 0.}, aR[4] = {0., 0., 0., 0.};
#pragma unroll
    for (int q = 0; q < 4; q++)
        aF[q] = da * ((jr ? lam_next[(size_t)q * n + j] : 0.0) - lam_next[(size_t)q * n + i]);
    StateDecisions D;
    bool ok;
    if (linear) {
        ok = states64_decide(A, C, 0.5 * dt, boost, gizmo, sl, sr, L, R, D);
    } else {
        ok = states64(A, C, 0.5 * dt, boost, false, false, L, R);
    }
    ok = ok && hll64_adj<HLLC>(L, R, nrm, A.w, C, boost, aF, aL, aR);
    if (ok && !linear) {
#pragma unroll
        for (int f = 0; f < 4; f++) {
            out[(size_t)f * F + m] = aL[f];
            out[(size_t)(4 + f) * F + m] = aR[f];
        }
#pragma unroll
        for (int r = 8; r < 24; r++) out[(size_t)r * F + m] = 0.;
    } else if (ok) {
        double asl[4], aol[4], asr[4], aor[4], agl[8], agr[8], rl, pl, rr, pr;
        side64_rev(aL, D.half_l, D.spat_l, gizmo, false, D, A.pi, A.gi, sl, sr, C.g, 0.5 * dt, asl, aol, agl, rl, pl, ok);
        side64_rev(aR, D.half_r, D.spat_r, gizmo, true, D, A.pj, A.gj, sr, sl, C.g, 0.5 * dt, asr, aor, agr, rr, pr, ok);
        if (ok) {
#pragma unroll
            for (int f = 0; f < 4; f++) {
                const double hi = f == 0 ? rl : (f == 3 ? pl : 0.), hj = f == 0 ? rr : (f == 3 ? pr : 0.);
                out[(size_t)f * F + m] = (asl[f] + hi) + aor[f];
                out[(size_t)(4 + f) * F + m] = (asr[f] + hj) + aol[f];
            }
#pragma unroll
            for (int r = 0; r < 8; r++) {
                out[(size_t)(8 + r) * F + m] = agl[r];
                out[(size_t)(16 + r) * F + m] = agr[r];
            }
        }
    }
    if (!ok) adj_face_plain(&M, &P, dt, prim, grad, face_w, lam_next, m, i, j, out);
}

// Sum of row x's face contributions (12 values: primitives, gradients), in list order.
__device__ __forceinline__ void gather_row(const phd_mesh &M, const double *face_adj, int x, double *s) {
    const int F = M.n_faces;
#pragma unroll
    for (int q = 0; q < 12; q++) s[q] = 0.0;
    for (int e = M.nbr_ptr[x]; e < M.nbr_ptr[x + 1]; e++) {
        const int f = M.nbr_idx[e];
        if (f < 0 || f >= F) continue;
        const bool as_i = M.pair_i[f] == x;
        const size_t pb = as_i ? 0 : 4, gb = as_i ? 8 : 16;
#pragma unroll
        for (int q = 0; q < 4; q++) s[q] += face_adj[(pb + q) * F + f];
#pragma unroll
        for (int q = 0; q < 8; q++) s[4 + q] += face_adj[(gb + q) * F + f];
    }
}

// Per real cell: its rows' face contributions (own and ghosts', with the reflective flips)
// and the reverse of the limited gradient (cell_gradient_f64): the primitives' part to
// prim_part, the neighbours' to entry_adj, the own one added to prim_part.  Ghost rows' entries
// get zeros (their gradient is their image's).  LINEAR: false for constant reconstruction,
// which has no gradients.
// The forward selections (unlimited estimate, limiter values, active entries, neighbour
// extrema) are recomputed here; k_adj_cell_taped reads them from the limiter record of a
// taped forward step.
// One kernel where a gather per cell, two clears and this reverse were four launches; the
// reverse's own arithmetic is fused multiply-adds on a reciprocal per entry (phd_fp64.cuh),
// 38 FP64 instructions an entry instead of 80.
template <bool LINEAR>
__global__ void __launch_bounds__(128) k_adj_cell(const __grid_constant__ phd_mesh M, phd_adj_index A, int limiter,
                                                  const double *__restrict__ prim, const double *face_adj,
                                                  double *__restrict__ entry_adj /* [4][2F] */,
                                                  double *__restrict__ prim_part /* [4][n] */) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= M.n_cells) return;
    pdl_wait();                                      // face_adj: the face kernel's
    const int n = M.n_cells, F = M.n_faces;
    const size_t E2 = 2 * (size_t)F;
    const int m0 = M.nbr_ptr[c], m1 = M.nbr_ptr[c + 1];
    double own[12];
    if (M.tag[c] != PHD_REAL_TAG) {
        gather_row(M, face_adj, c, own);             // the primitives' part, folded by k_adj_final
#pragma unroll
        for (int f = 0; f < 4; f++) prim_part[(size_t)f * n + c] = own[f];
        if (LINEAR)
            for (int e = m0; e < m1; e++)
#pragma unroll
                for (int f = 0; f < 4; f++) entry_adj[f * E2 + e] = 0.0;
        return;
    }
    gather_row(M, face_adj, c, own);
    if (!LINEAR) {
#pragma unroll
        for (int f = 0; f < 4; f++) prim_part[(size_t)f * n + c] = own[f];
        return;
    }
    // lam_grad of this cell = own row + its ghost rows (reflective diagonal flip)
    double *ag = own + 4;
    for (int t = A.ghost_ptr[c]; t < A.ghost_ptr[c + 1]; t++) {
        const int g = A.ghost_idx[t];
        const int fl = M.flip ? M.flip[g] : 0;
        double row[12];
        gather_row(M, face_adj, g, row);
        if (fl & 1) row[6] = -row[6];
        if (fl & 2) row[9] = -row[9];
#pragma unroll
        for (int q = 0; q < 8; q++) ag[q] += row[4 + q];
    }
    double xi[2], cx[2], pc[4], df[8], alpha[4] = {1.0, 1.0, 1.0, 1.0};
    int arg_max[4], arg_min[4];
    int act[4] = {-1, -1, -1, -1};     // entry whose psi is the active limit
    int act_f0 = -1;                   // TESS: field of the active psi
    for (int k = 0; k < 2; k++) {
        xi[k] = M.x[(size_t)k * n + c];
        cx[k] = xi[k] + M.dcom[(size_t)k * n + c];
    }
    const double vol = M.vol[c];
    // forward recompute (cell_gradient_f64 with selections)
    double phi_max[4], phi_min[4];
    for (int f = 0; f < 4; f++) {
        pc[f] = prim[(size_t)f * n + c];
        phi_max[f] = phi_min[f] = pc[f];
        arg_max[f] = arg_min[f] = -1;
        df[2 * f] = df[2 * f + 1] = 0.0;
    }
    for (int e = m0; e < m1; e++) {
        const int fid = M.nbr_idx[e];
        const int j = (M.pair_i[fid] == c) ? M.pair_j[fid] : M.pair_i[fid];
        const double area = M.area[fid];
        double cfx[2], dr[2], r = 0.0;
        for (int k = 0; k < 2; k++) {
            const double xj = M.x[(size_t)k * n + j];
            cfx[k] = M.com[(size_t)k * F + fid] - 0.5 * (xi[k] + xj);
            dr[k] = xi[k] - xj;
            r = r + t_sq(dr[k]);
        }
        r = sqrt(r);
        for (int f = 0; f < 4; f++) {
            const double pj = prim[(size_t)f * n + j];
            if (pj > phi_max[f]) { phi_max[f] = pj; arg_max[f] = e; }
            if (pj < phi_min[f]) { phi_min[f] = pj; arg_min[f] = e; }
            const double d_dif = pj - pc[f], d_sum = pj + pc[f];
            for (int k = 0; k < 2; k++)
                df[2 * f + k] = df[2 * f + k] + (area * ((d_dif * cfx[k]) - ((0.5 * d_sum) * dr[k]))) / (r * vol);
        }
    }
    for (int e = m0; e < m1; e++) {
        const int fid = M.nbr_idx[e];
        const int j = (M.pair_i[fid] == c) ? M.pair_j[fid] : M.pair_i[fid];
        double sep[2];
        for (int k = 0; k < 2; k++) sep[k] = M.com[(size_t)k * F + fid] - cx[k];
        for (int f = 0; f < 4; f++) {
            double dphi = 0.0, psi;
            for (int k = 0; k < 2; k++) dphi = dphi + df[2 * f + k] * sep[k];
            if (limiter == PHD_LIMITER_AREPO) {
                if (dphi > 0) psi = (phi_max[f] - pc[f]) / dphi;
                else if (dphi < 0) psi = (phi_min[f] - pc[f]) / dphi;
                else psi = 1.0;
                const double cand = fmax(psi, 0.);
                if (cand < alpha[f]) { alpha[f] = cand; act[f] = (psi > 0.0 && dphi != 0.0) ? e : -2; }
            } else {
                if (dphi > 0.0 || dphi < 0.0) {
                    const double t = (prim[(size_t)f * n + j] - pc[f]) / dphi;
                    psi = (0. > t) ? 0. : t;
                } else psi = 1.0;
                const double cand = fmax(psi, 0.);
                if (cand < alpha[0]) { alpha[0] = cand; act[0] = (psi > 0.0 && dphi != 0.0) ? e : -2; act_f0 = f; }
            }
        }
    }
    // reverse: grad = alpha * df
    double adf[8], aself[4] = {0, 0, 0, 0}, aalpha[4];
#pragma unroll
    for (int f = 0; f < 4; f++) {
        aalpha[f] = fma(df[2 * f], ag[2 * f], df[2 * f + 1] * ag[2 * f + 1]);
        adf[2 * f] = alpha[f] * ag[2 * f];
        adf[2 * f + 1] = alpha[f] * ag[2 * f + 1];
    }
    // limiter: active psi -> (extreme value, own value, df)
    double aext[4] = {0, 0, 0, 0};       // adjoint of the active entry's phi_max / phi_min (TESS: neighbour)
    int ext[4] = {-1, -1, -1, -1};       // and the entry it belongs to (-1: the cell itself)
    const bool tess = limiter == PHD_LIMITER_TESS;
#pragma unroll
    for (int f = 0; f < 4; f++) {
        const int e = act[f];
        if (e < 0 || (tess && f != 0)) continue;
        const int ff = tess ? act_f0 : f, fid = M.nbr_idx[e];
        const double s0 = M.com[fid] - cx[0], s1 = M.com[(size_t)F + fid] - cx[1];
        double d0 = df[2 * f], d1 = df[2 * f + 1];
        if (tess) {
#pragma unroll
            for (int g = 0; g < 4; g++) { d0 = g == ff ? df[2 * g] : d0; d1 = g == ff ? df[2 * g + 1] : d1; }
        }
        const double dphi = d0 * s0 + d1 * s1;
        bool ok = true;
        double y = f64_rcp(dphi, ok);
        if (!ok) y = 1.0 / dphi;
        const double ap = aalpha[f] * y, ad = -ap * alpha[f];
        const int arg = tess ? e : (f64_pos(dphi) ? arg_max[f] : arg_min[f]);
#pragma unroll
        for (int g = 0; g < 4; g++)
            if (g == ff) {
                adf[2 * g] = fma(ad, s0, adf[2 * g]);
                adf[2 * g + 1] = fma(ad, s1, adf[2 * g + 1]);
                aself[g] -= ap;
                if (arg >= 0) {
                    aext[g] = ap;
                    ext[g] = arg;
                } else {
                    aself[g] += ap;
                }
            }
    }
    // df = sum_e area (d_dif cfx - d_sum dr / 2) / (r vol)
    for (int e = m0; e < m1; e++) {
        const int fid = M.nbr_idx[e];
        const int j = (M.pair_i[fid] == c) ? M.pair_j[fid] : M.pair_i[fid];
        const double area = M.area[fid];
        const double xj = M.x[j], yj = M.x[(size_t)n + j];
        const double cfx = fma(-0.5, xi[0] + xj, M.com[fid]), cfy = fma(-0.5, xi[1] + yj, M.com[(size_t)F + fid]);
        const double dx = xi[0] - xj, dy = xi[1] - yj;
        bool ok = true;
        double r2 = fma(dx, dx, dy * dy), r = f64_sqrt(r2, ok), y = f64_rcp(r * vol, ok);
        if (!ok) {
            r = sqrt(r2);
            y = 1.0 / (r * vol);
        }
        const double coef = area * y;
        const double jx = coef * fma(-0.5, dx, cfx), jy = coef * fma(-0.5, dy, cfy);      // d df / d phi_j
        const double sx = -coef * fma(0.5, dx, cfx), sy = -coef * fma(0.5, dy, cfy);      // d df / d phi_c
#pragma unroll
        for (int f = 0; f < 4; f++) {
            double aj = fma(adf[2 * f], jx, adf[2 * f + 1] * jy);
            aself[f] = fma(adf[2 * f], sx, fma(adf[2 * f + 1], sy, aself[f]));
            if (ext[f] == e) aj += aext[f];
            entry_adj[f * E2 + e] = aj;
        }
    }
#pragma unroll
    for (int f = 0; f < 4; f++) prim_part[(size_t)f * n + c] = own[f] + aself[f];
}

// Row x's sums of field f's face contributions (the primitive's, the gradient's two), in list
// order, the loads of four faces at a time.
__device__ __forceinline__ void gather_field(const phd_mesh &M, const double *face_adj, int x, int f,
                                             double &s0, double &s1, double &s2) {
    const int F = M.n_faces, m0 = M.nbr_ptr[x], m1 = M.nbr_ptr[x + 1];
    s0 = s1 = s2 = 0.0;
    constexpr int CH = 4;
    for (int eb = m0; eb < m1; eb += CH) {
        int fid[CH];
        double v[CH][3];
#pragma unroll
        for (int k = 0; k < CH; k++) fid[k] = eb + k < m1 ? M.nbr_idx[eb + k] : -1;
#pragma unroll
        for (int k = 0; k < CH; k++) {
            v[k][0] = v[k][1] = v[k][2] = 0.0;
            if (fid[k] < 0 || fid[k] >= F) continue;
            const bool as_i = M.pair_i[fid[k]] == x;
            const size_t pb = as_i ? 0 : 4, gb = as_i ? 8 : 16;
            v[k][0] = face_adj[(pb + f) * F + fid[k]];
            v[k][1] = face_adj[(gb + 2 * f) * F + fid[k]];
            v[k][2] = face_adj[(gb + 2 * f + 1) * F + fid[k]];
        }
#pragma unroll
        for (int k = 0; k < CH; k++) {
            if (fid[k] < 0 || fid[k] >= F) continue;
            s0 += v[k][0];
            s1 += v[k][1];
            s2 += v[k][2];
        }
    }
}

// k_adj_cell<true> after a taped forward step, by four threads a cell, each with one field: the
// gathered sums and the limiter's reverse are its own, the lists' geometry is formed by one
// thread an entry and handed round.  A thread a cell left three or four warps on an SM, each
// with 415 FP64 instructions one behind the other (16,384 cells: 35.4 -> 23.5 us); the sums
// keep their order.
__global__ void __launch_bounds__(128) k_adj_cell_taped(const __grid_constant__ phd_mesh M, phd_adj_index A, int limiter,
                                                        const double *face_adj,
                                                        double *__restrict__ entry_adj, double *__restrict__ prim_part,
                                                        const double *__restrict__ tape_f64,
                                                        const int32_t *__restrict__ tape_i32) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, c = t >> 2, f = t & 3;
    if (c >= M.n_cells) return;                      // whole quads
    const unsigned quad = 0xfu << (threadIdx.x & 28);
    const int n = M.n_cells, F = M.n_faces;
    const size_t E2 = 2 * (size_t)F;
    const int m0 = M.nbr_ptr[c], m1 = M.nbr_ptr[c + 1];
    const bool real = M.tag[c] == PHD_REAL_TAG;
    const double xc = M.x[c], yc = M.x[(size_t)n + c], cx = xc + M.dcom[c], cy = yc + M.dcom[(size_t)n + c];
    const double vol = M.vol[c];
    const double df0 = tape_f64[(size_t)(2 * f) * n + c], df1 = tape_f64[(size_t)(2 * f + 1) * n + c];
    const double alpha = tape_f64[(size_t)(8 + f) * n + c];
    int act = tape_i32[(size_t)f * n + c], ff = f;
    pdl_wait();                                      // face_adj: the face kernel's
    double own, ag0, ag1;
    gather_field(M, face_adj, c, f, own, ag0, ag1);
    if (!real) {
        prim_part[(size_t)f * n + c] = own;          // the primitives' part, folded by k_adj_final
        for (int e = m0; e < m1; e++) entry_adj[f * E2 + e] = 0.0;
        return;
    }
    for (int g = A.ghost_ptr[c]; g < A.ghost_ptr[c + 1]; g++) {
        const int x = A.ghost_idx[g], fl = M.flip ? M.flip[x] : 0;
        double s0, s1, s2;
        gather_field(M, face_adj, x, f, s0, s1, s2);
        ag0 += (f == 1 && (fl & 1)) ? -s1 : s1;
        ag1 += (f == 2 && (fl & 2)) ? -s2 : s2;
    }
    const bool tess = limiter == PHD_LIMITER_TESS;
    // reverse: grad = alpha * df
    double adf0 = alpha * ag0, adf1 = alpha * ag1, aself = 0.0, aext = 0.0;
    int ext = -1;                                    // the entry aext belongs to
    // limiter: active psi -> (extreme value, own value, df); with TESS the density's, whose
    // entry's ratio is that of field ff
    double aalpha = fma(df0, ag0, df1 * ag1), al = alpha, d0 = df0, d1 = df1;
    if (tess) {
        act = __shfl_sync(quad, act, 0, 4);
        ff = act >= 0 ? tape_i32[(size_t)12 * n + c] : 0;
        aalpha = __shfl_sync(quad, aalpha, 0, 4);
        al = __shfl_sync(quad, alpha, 0, 4);
        d0 = __shfl_sync(quad, df0, ff, 4);
        d1 = __shfl_sync(quad, df1, ff, 4);
    }
    if (act >= 0 && ff == f) {
        const int fid = M.nbr_idx[act];
        const double s0 = M.com[fid] - cx, s1 = M.com[(size_t)F + fid] - cy;
        const double dphi = d0 * s0 + d1 * s1;
        bool ok = true;
        double y = f64_rcp(dphi, ok);
        if (!ok) y = 1.0 / dphi;
        const double ap = aalpha * y, ad = -ap * al;
        const int arg = tess ? act : tape_i32[(size_t)((f64_pos(dphi) ? 4 : 8) + f) * n + c];
        adf0 = fma(ad, s0, adf0);
        adf1 = fma(ad, s1, adf1);
        if (arg >= 0) {
            aself -= ap;
            aext = ap;
            ext = arg;
        }
    }
    // df = sum_e area (d_dif cfx - d_sum dr / 2) / (r vol)
    for (int eb = m0; eb < m1; eb += 4) {
        const int fid = M.nbr_idx[min(eb + f, m1 - 1)];
        const int j = (M.pair_i[fid] == c) ? M.pair_j[fid] : M.pair_i[fid];
        const double area = M.area[fid];
        const double xj = M.x[j], yj = M.x[(size_t)n + j];
        const double cfx = fma(-0.5, xc + xj, M.com[fid]), cfy = fma(-0.5, yc + yj, M.com[(size_t)F + fid]);
        const double dx = xc - xj, dy = yc - yj;
        bool ok = true;
        double r2 = fma(dx, dx, dy * dy), r = f64_sqrt(r2, ok), y = f64_rcp(r * vol, ok);
        if (!ok) {
            r = sqrt(r2);
            y = 1.0 / (r * vol);
        }
        const double coef = area * y;
        const double jx = coef * fma(-0.5, dx, cfx), jy = coef * fma(-0.5, dy, cfy);      // d df / d phi_j
        const double sx = -coef * fma(0.5, dx, cfx), sy = -coef * fma(0.5, dy, cfy);      // d df / d phi_c
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (eb + k >= m1) break;                 // uniform over the quad
            const double Jx = __shfl_sync(quad, jx, k, 4), Jy = __shfl_sync(quad, jy, k, 4);
            const double Sx = __shfl_sync(quad, sx, k, 4), Sy = __shfl_sync(quad, sy, k, 4);
            double aj = fma(adf0, Jx, adf1 * Jy);
            aself = fma(adf0, Sx, fma(adf1, Sy, aself));
            if (ext == eb + k) aj += aext;
            entry_adj[f * E2 + eb + k] = aj;
        }
    }
    prim_part[(size_t)f * n + c] = own + aself;
}

// Per real cell: its rows' primitive adjoints (own and ghosts', flipped) with the neighbours'
// gradient parts, through the primitive recovery, plus the identity of the update; ghost
// rows of lam are zero.
template <bool LINEAR>
__global__ void __launch_bounds__(128) k_adj_final(const __grid_constant__ phd_mesh M, phd_adj_index A, double gamma,
                                                   const double *__restrict__ cons, const double *prim_part,
                                                   const double *entry_adj,
                                                   const double *__restrict__ lam_next, double *__restrict__ lam) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= M.n_cells) return;
    const int n = M.n_cells;
    const size_t E2 = 2 * (size_t)M.n_faces;
    if (M.tag[c] != PHD_REAL_TAG) {
        for (int q = 0; q < 4; q++) lam[(size_t)q * n + c] = 0.0;
        return;
    }
    double ap[4] = {0., 0., 0., 0.};
    const int t0 = A.ghost_ptr[c], t1 = A.ghost_ptr[c + 1];
    const double m = cons[c], mx = cons[(size_t)n + c], my = cons[2 * (size_t)n + c], vol = M.vol[c];
    pdl_wait();                                      // prim_part, entry_adj: the cell kernel's
    for (int t = t0 - 1; t < t1; t++) {              // the cell itself, then its ghosts
        const int x = t < t0 ? c : A.ghost_idx[t];
        const int fl = (t >= t0 && M.flip) ? M.flip[x] : 0;
        double s[4];
#pragma unroll
        for (int f = 0; f < 4; f++) s[f] = prim_part[(size_t)f * n + x];
        if (LINEAR) {
            for (int e = M.nbr_ptr[x]; e < M.nbr_ptr[x + 1]; e++) {
                const int pe = A.partner[e];
                if (pe < 0 || (size_t)pe >= E2) continue;
#pragma unroll
                for (int f = 0; f < 4; f++) s[f] += entry_adj[f * E2 + pe];
            }
        }
        if (fl & 1) s[1] = -s[1];
        if (fl & 2) s[2] = -s[2];
#pragma unroll
        for (int f = 0; f < 4; f++) ap[f] += s[f];
    }
    bool ok = true;
    double im = f64_rcp(m, ok), iv = f64_rcp(vol, ok);
    if (!ok) {
        im = 1.0 / m;
        iv = 1.0 / vol;
    }
    const double rho = m * iv, vx = mx * im, vy = my * im;
    const double g1 = gamma - 1.0, a3 = ap[3] * g1;
    // p = (E/V - rho v^2 / 2)(gamma - 1)
    const double arho = fma(-0.5 * a3, fma(vx, vx, vy * vy), ap[0]);
    const double ax = fma(-a3 * rho, vx, ap[1]) * im, ay = fma(-a3 * rho, vy, ap[2]) * im;
    lam[c] = lam_next[c] + fma(arho, iv, -fma(ax, vx, ay * vy));
    lam[(size_t)n + c] = lam_next[(size_t)n + c] + ax;
    lam[2 * (size_t)n + c] = lam_next[2 * (size_t)n + c] + ay;
    lam[3 * (size_t)n + c] = lam_next[3 * (size_t)n + c] + a3 * iv;
}

inline int ba(int n) { return block_for(n, BA); }
inline int ga(int n) { return grid_for_block(n, ba(n)); }

}  // namespace phd

using namespace phd;

extern "C" {

static int adjoint_step(const phd_mesh *mesh, const phd_adj_index *index, const phd_params *par, double dt,
                        const double *cons, const double *prim, const double *grad, const double *face_w,
                        const double *lam_next, double *lam, double *work, const double *tape_f64,
                        const int32_t *tape_i32, cudaStream_t stream);

int phd_adjoint_step_f64(const phd_mesh *mesh, const phd_adj_index *index, const phd_params *par, double dt,
                         const double *cons, const double *prim, const double *grad, const double *face_w,
                         const double *lam_next, double *lam, double *work, cudaStream_t stream) {
    phd::NvtxRange nvtx_range("phd_adjoint_step_f64");
    return adjoint_step(mesh, index, par, dt, cons, prim, grad, face_w, lam_next, lam, work, nullptr, nullptr,
                        stream);
}

int phd_adjoint_step_f64_taped(const phd_mesh *mesh, const phd_adj_index *index, const phd_params *par,
                               double dt, const double *cons, const double *prim, const double *grad,
                               const double *face_w, const double *lam_next, double *lam, double *work,
                               const double *tape_f64, const int32_t *tape_i32, cudaStream_t stream) {
    phd::NvtxRange nvtx_range("phd_adjoint_step_f64_taped");
    if (!tape_f64 || !tape_i32) return PHD_ERR_ARG;
    return adjoint_step(mesh, index, par, dt, cons, prim, grad, face_w, lam_next, lam, work, tape_f64, tape_i32,
                        stream);
}

static int adjoint_step(const phd_mesh *mesh, const phd_adj_index *index, const phd_params *par, double dt,
                        const double *cons, const double *prim, const double *grad, const double *face_w,
                        const double *lam_next, double *lam, double *work, const double *tape_f64,
                        const int32_t *tape_i32, cudaStream_t stream) {
    if (!mesh || mesh->dim != 2 || !index || !par || !cons || !prim || !lam_next || !lam || !work)
        return PHD_ERR_ARG;
    if (mesh->n_faces && !mesh->normal) return PHD_ERR_ARG;
    if (par->solver < PHD_HLL || par->solver > PHD_EXACT) return PHD_ERR_ARG;
    if (par->reconstruction == PHD_LINEAR && !grad) return PHD_ERR_ARG;
    const phd_mesh &M = *mesh;
    const size_t n = M.n_cells, F = M.n_faces;
    double *face_adj = work;                       // [24][F]
    double *entry_adj = face_adj + 24 * F;         // [4][2F]
    double *prim_part = entry_adj + 8 * F;         // [4][n]
    // the first kernel waits for the stream, the others come in behind each other
    PdlQueue queue = {stream};
    if (F && par->solver == PHD_EXACT)
        launch_pdl(k_adj_face_exact, ga((int)F), ba((int)F), queue, M, *par, dt, prim, grad, face_w, lam_next, face_adj);
    else if (F) {
        const int block = (int)F < 16 * 128 * sm_count_current() ? 32 : 128, grid = grid_for_block((int)F, block);
        const Gas64 C = gas64(par->gamma);
        if (par->solver == PHD_HLLC)
            launch_pdl(k_adj_face<true>, grid, block, queue, M, *par, C, dt, prim, grad, face_w, lam_next, face_adj);
        else
            launch_pdl(k_adj_face<false>, grid, block, queue, M, *par, C, dt, prim, grad, face_w, lam_next, face_adj);
    }
    const int bc = block_for((int)n, 128), gc = grid_for_block((int)n, bc);
    if (par->reconstruction != PHD_LINEAR) {
        launch_pdl(k_adj_cell<false>, gc, bc, queue, M, *index, par->limiter, prim, face_adj, entry_adj, prim_part);
        launch_pdl(k_adj_final<false>, gc, bc, queue, M, *index, par->gamma, cons, prim_part, entry_adj, lam_next, lam);
    } else {
        if (tape_f64) {
            const int bt = block_for(4 * (int)n, 128);
            launch_pdl(k_adj_cell_taped, grid_for_block(4 * (int)n, bt), bt, queue, M, *index, par->limiter, face_adj,
                       entry_adj, prim_part, tape_f64, tape_i32);
        } else {
            launch_pdl(k_adj_cell<true>, gc, bc, queue, M, *index, par->limiter, prim, face_adj, entry_adj, prim_part);
        }
        launch_pdl(k_adj_final<true>, gc, bc, queue, M, *index, par->gamma, cons, prim_part, entry_adj, lam_next, lam);
    }
    return cudaPeekAtLastError() == cudaSuccess ? PHD_OK : PHD_ERR_LAUNCH;
}

size_t phd_adjoint_work_doubles(int32_t n_cells, int32_t n_faces) {
    return (size_t)24 * n_faces + 12 * (size_t)n_cells + 8 * (size_t)n_faces + 8 * (size_t)n_cells;
}

}  // extern "C"

// ---- adjoint step that allocates nothing --------------------------------------------
// Work space for phd_adjoint_step_f64_noalloc: a fixed array in the library's device
// image, created on every GPU where the library is loaded and kept until the process
// exits.  Its size is the limit of that entry point (PHD_ADJ_NOALLOC_MAX_DOUBLES).
static __device__ __align__(256) double g_adj_scratch[PHD_ADJ_NOALLOC_MAX_DOUBLES];

namespace {

// Device address of g_adj_scratch in the current device's current context.  In host
// code the symbol name is only a host-side stand-in, so the address is asked from the
// runtime on every call (cheap once the library's device code is loaded there): a
// cached address would go stale after cudaDeviceReset, or point into the wrong module
// when the caller switches contexts.
double *adj_scratch_on_current_device(int *rc) {
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_adj_scratch);
    if (e != cudaSuccess || !p) {
        *rc = PHD_ERR_LAUNCH;
        return nullptr;
    }
    return static_cast<double *>(p);
}

}  // namespace

extern "C" {

int phd_adjoint_step_f64_noalloc(const phd_mesh *mesh, const phd_adj_index *index, const phd_params *par,
                                 double dt, const double *cons, const double *prim, const double *grad,
                                 const double *face_w, const double *lam_next, double *lam, cudaStream_t stream) {
    phd::NvtxRange nvtx_range("phd_adjoint_step_f64_noalloc");
    if (!mesh || mesh->n_cells < 0 || mesh->n_faces < 0) return PHD_ERR_ARG;
    if (phd_adjoint_work_doubles(mesh->n_cells, mesh->n_faces) > (size_t)PHD_ADJ_NOALLOC_MAX_DOUBLES)
        return PHD_ERR_SCRATCH_TOO_SMALL;
    int rc = PHD_OK;
    double *work = adj_scratch_on_current_device(&rc);
    if (!work) return rc;
    return phd_adjoint_step_f64(mesh, index, par, dt, cons, prim, grad, face_w, lam_next, lam, work, stream);
}

}  // extern "C"
