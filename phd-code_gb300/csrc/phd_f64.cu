// phd_f64.cu -- FP64 kernels: one per reference plugin stage, plus the fused step.
//
// Compiled with --fmad=false: every product and sum rounds separately, as in the
// reference's Cython build, so results match the reference to the last few ulps
// (only CUDA's pow/sqrt library rounding can differ from libm's).
#include "phd_common.cuh"
#include "phd_physics.cuh"
#include "phd_ref.cuh"
#include "phd_face64.cuh"
#include "phd_exact64.cuh"

namespace phd {

constexpr int BLOCK = 256;

__device__ __forceinline__ void set_status(phd_clock *clk, int bits) {
    if (bits && clk) atomicOr(&clk->status, bits);
}

// ---- gradients ------------------------------------------------------------------
// Limiter record of one cell's gradient, kept by a taped forward step for the adjoint:
// f64 [12][n]: the unlimited estimate (8 rows) and the limiter values (4 rows);
// i32 [13][n]: per field the CSR entry of the active limit (-1: none, -2: a clamp at
// zero or a flat field), the entries of the neighbour maximum and minimum (-1: the
// cell itself), and (TESS) the field of the active limit.
struct GradTape {
    double *f64;
    int32_t *i32;
};

// PieceWiseLinear.compute_gradients reconstruction.pyx:620-736 for cell c, result in
// df (limited).  Returns status bits.  TAPE: also records the limiter's selections
// (same arithmetic; only bookkeeping is added) when `record`.
template <int DIM, bool TAPE = false>
__device__ int cell_gradient_f64(const phd_mesh &M, const double *prim, int limiter,
                                 int c, double *df, GradTape tape = GradTape{nullptr, nullptr},
                                 bool record = false) {
    constexpr int NF = DIM + 2;
    const int n = M.n_cells, F = M.n_faces;
    double phi_max[NF], phi_min[NF], alpha[NF], xi[DIM], cx[DIM], pc[NF];
    int arg_max[NF], arg_min[NF], act[NF], act_f0 = -1;
    int status = 0;
#pragma unroll
    for (int k = 0; k < DIM; k++) {
        xi[k] = M.x[(size_t)k * n + c];
        cx[k] = xi[k] + M.dcom[(size_t)k * n + c];
    }
    const double vol = M.vol[c];
#pragma unroll
    for (int f = 0; f < NF; f++) {
        pc[f] = prim[(size_t)f * n + c];
        phi_max[f] = phi_min[f] = pc[f];
        alpha[f] = 1.0;
        arg_max[f] = arg_min[f] = act[f] = -1;
#pragma unroll
        for (int k = 0; k < DIM; k++) df[DIM * f + k] = 0;
    }
    const int m0 = M.nbr_ptr[c], m1 = M.nbr_ptr[c + 1];
    for (int m = m0; m < m1; m++) {
        const int fid = M.nbr_idx[m];
        if (fid < 0 || fid >= F) { status |= PHD_STATUS_BAD_INDEX; continue; }
        const double area = M.area[fid];
        int j;
        const int a = M.pair_i[fid], b = M.pair_j[fid];
        if (c == a) j = b;
        else if (c == b) j = a;
        else { status |= PHD_STATUS_BAD_INDEX; continue; }
        if (j < 0 || j >= n) { status |= PHD_STATUS_BAD_INDEX; continue; }
        double cfx[DIM], dr[DIM], r = 0.0;
#pragma unroll
        for (int k = 0; k < DIM; k++) {
            const double xj = M.x[(size_t)k * n + j];
            cfx[k] = M.com[(size_t)k * F + fid] - 0.5 * (xi[k] + xj);
            dr[k] = xi[k] - xj;
            r = r + t_sq(dr[k]);
        }
        r = sqrt(r);
#pragma unroll
        for (int f = 0; f < NF; f++) {
            const double pj = prim[(size_t)f * n + j];
            if (TAPE) {
                if (pj > phi_max[f]) arg_max[f] = m;
                if (pj < phi_min[f]) arg_min[f] = m;
            }
            phi_max[f] = fmax(phi_max[f], pj);
            phi_min[f] = fmin(phi_min[f], pj);
            const double d_dif = pj - pc[f];
            const double d_sum = pj + pc[f];
#pragma unroll
            for (int k = 0; k < DIM; k++)
                df[DIM * f + k] = df[DIM * f + k] + (area * ((d_dif * cfx[k]) - ((0.5 * d_sum) * dr[k]))) / (r * vol);
        }
    }
    if (limiter == PHD_LIMITER_AREPO) {
        for (int m = m0; m < m1; m++) {
            const int fid = M.nbr_idx[m];
            if (fid < 0 || fid >= F) continue;
            double sep[DIM];
#pragma unroll
            for (int k = 0; k < DIM; k++) sep[k] = M.com[(size_t)k * F + fid] - cx[k];
#pragma unroll
            for (int f = 0; f < NF; f++) {
                double dphi = 0.0, psi;
#pragma unroll
                for (int k = 0; k < DIM; k++) dphi = dphi + df[DIM * f + k] * sep[k];
                if (dphi > 0) psi = (phi_max[f] - pc[f]) / dphi;
                else if (dphi < 0) psi = (phi_min[f] - pc[f]) / dphi;
                else psi = 1.0;
                if (TAPE && fmax(psi, 0.) < alpha[f]) act[f] = (psi > 0.0 && dphi != 0.0) ? m : -2;
                alpha[f] = fmin(alpha[f], fmax(psi, 0.));
            }
        }
    } else if (limiter == PHD_LIMITER_TESS) {
        for (int m = m0; m < m1; m++) {
            const int fid = M.nbr_idx[m];
            if (fid < 0 || fid >= F) continue;
            const int a = M.pair_i[fid], b = M.pair_j[fid];
            const int j = (c == a) ? b : a;
            if (j < 0 || j >= n) continue;
            double sep[DIM];
#pragma unroll
            for (int k = 0; k < DIM; k++) sep[k] = M.com[(size_t)k * F + fid] - cx[k];
#pragma unroll
            for (int f = 0; f < NF; f++) {
                double dphi = 0.0, psi;
#pragma unroll
                for (int k = 0; k < DIM; k++) dphi = dphi + df[DIM * f + k] * sep[k];
                if (dphi > 0.0 || dphi < 0.0) {
                    const double t = (prim[(size_t)f * n + j] - pc[f]) / dphi;
                    psi = (0. > t) ? 0. : t;
                } else psi = 1.0;
                if (TAPE && fmax(psi, 0.) < alpha[0]) {
                    act[0] = (psi > 0.0 && dphi != 0.0) ? m : -2;
                    act_f0 = f;
                }
                alpha[0] = fmin(alpha[0], fmax(psi, 0.));     // only alpha[0]: :731
            }
        }
    }
    if (TAPE && record) {
#pragma unroll
        for (int r = 0; r < NF * DIM; r++) tape.f64[(size_t)r * n + c] = df[r];
#pragma unroll
        for (int f = 0; f < NF; f++) {
            tape.f64[(size_t)(NF * DIM + f) * n + c] = alpha[f];
            tape.i32[(size_t)f * n + c] = act[f];
            tape.i32[(size_t)(NF + f) * n + c] = arg_max[f];
            tape.i32[(size_t)(2 * NF + f) * n + c] = arg_min[f];
        }
        tape.i32[(size_t)(3 * NF) * n + c] = act_f0;
    }
#pragma unroll
    for (int f = 0; f < NF; f++)
#pragma unroll
        for (int k = 0; k < DIM; k++) df[DIM * f + k] = alpha[f] * df[DIM * f + k];
    return status;
}

// Mesh.assign_generator_velocities mesh.pyx:397-426 for cell i on the plain path.
__device__ __noinline__ void generator_velocity_plain(const phd_mesh *M, const double *prim, double gamma, double eta,
                                                      int regularize, int i, double *wx) {
    const int n = M->n_cells;
#pragma unroll
    for (int k = 0; k < 2; k++) wx[k] = prim[(size_t)(1 + k) * n + i];
    if (regularize) {
        const double c = sqrt((gamma * prim[(size_t)3 * n + i]) / prim[i]);
        double d = 0.0;
#pragma unroll
        for (int k = 0; k < 2; k++) d = d + t_sq(M->dcom[(size_t)k * n + i]);
        d = sqrt(d);
        const double R = sqrt(M->vol[i] / 3.141592653589793);
        if ((0.9 <= (d / (eta * R))) && ((d / (eta * R)) < 1.1)) {
#pragma unroll
            for (int k = 0; k < 2; k++)
                wx[k] = wx[k] + (((c * M->dcom[(size_t)k * n + i]) * (d - ((0.9 * eta) * R))) / (((d * 0.2) * eta) * R));
        } else if (1.1 <= (d / (eta * R))) {
#pragma unroll
            for (int k = 0; k < 2; k++) wx[k] = wx[k] + ((c * M->dcom[(size_t)k * n + i]) / d);
        }
    }
}

// The same numbers with seeded quotients and roots; the sound speed only where a cell is off
// its centroid far enough to be steered.
__device__ __forceinline__ void generator_velocity(const phd_mesh &M, const double *prim, double gamma,
                                                   double eta, int regularize, int i, double *__restrict__ w) {
    const int n = M.n_cells;
    double wx[2] = {prim[(size_t)n + i], prim[2 * (size_t)n + i]};
    if (regularize) {
        bool ok = true;
        const double dc[2] = {M.dcom[i], M.dcom[(size_t)n + i]};
        const double d2 = dc[0] * dc[0] + dc[1] * dc[1];
        const double eR = eta * f64_sqrt(f64_div_by(M.vol[i], 3.141592653589793, 1.0 / 3.141592653589793, ok), ok);
        double d = 0.0, q = 0.0;
        if (!f64_zero(d2)) {
            d = f64_sqrt(d2, ok);
            q = f64_div(d, eR, ok);
        } else {
            f64_rcp(eR, ok);                         // eta R within the window, as with d > 0
        }
        if (f64_le(0.9, q)) {
            const double c = f64_sqrt(f64_div(gamma * prim[3 * (size_t)n + i], prim[i], ok), ok);
            double num = 1.0, den = d;
            if (f64_lt(q, 1.1)) {
                const double R = f64_sqrt(f64_div_by(M.vol[i], 3.141592653589793, 1.0 / 3.141592653589793, ok), ok);
                num = d - (0.9 * eta) * R;
                den = ((d * 0.2) * eta) * R;
            }
            const double y = f64_rcp(den, ok);
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const double cd = c * dc[k];
                wx[k] = wx[k] + f64_div_by(f64_lt(q, 1.1) ? cd * num : cd, den, y, ok);
            }
        }
        if (!ok) generator_velocity_plain(&M, prim, gamma, eta, regularize, i, wx);
    }
    w[i] = wx[0];
    w[(size_t)n + i] = wx[1];
}

// One row of the gradient on the plain path: a real cell's own gradient, a ghost's its
// image's (computed again from the image's faces, bit-identical) with the reflective
// diagonal flip of grad v (domain_manager.pyx:819-835, boundary.pyx:287-307).
template <bool TAPE>
__device__ __noinline__ int gradient_row_plain(const phd_mesh *M, const double *prim, int limiter, int i, int c,
                                               double *grad, GradTape tape) {
    double df[8];
    const int st = cell_gradient_f64<2, TAPE>(*M, prim, limiter, c, df, tape, i == c);
    const int fl = M->flip ? M->flip[i] : 0;
    if (fl & 1) df[2] *= -1;
    if (fl & 2) df[5] *= -1;
#pragma unroll
    for (int r = 0; r < 8; r++) grad[(size_t)r * M->n_cells + i] = df[r];
    return st;
}

// The step's kernels are launched with programmatic stream serialization (PdlQueue): a kernel's
// blocks come in as the last ones of the kernel before leave, do what concerns the mesh alone
// (row setup and lists here, geometry and list heads in the face and update kernels) and wait
// only then.  Measured against plain launches: 10,000 cells 64 -> 57 us a step, 66,000 240 ->
// 232, 40 adjoint steps at 128 x 128 9.85 -> 9.5 ms.  Letting them in earlier (launch_dependents on
// entry) puts most of them on the SMs that happen to be free: 75 us a step at 10,000 cells.

// Limited gradients of NC rows (cells) by 4 NC threads, the same numbers as cell_gradient_f64
// bit for bit.  The kernel is bound by the FP64 pipe (phd_fp64.cuh), so the work is laid
// out for few and full FP64 warp instructions:
//  * per face of the block, one thread forms the face's terms of the Green-Gauss sum for
//    both of its cells: the numerators area (d_dif c - d_sum dr / 2) differ only in sign
//    between the two sides, the quotients by r V take one seed a side.  (A thread a cell
//    formed every numerator twice, and its warp ran as long as its longest list: 20 of 32
//    lanes active.)  Where the other cell lies outside the block its side is left out, and
//    such faces are kept apart from the others so that their warps skip it too;
//  * the terms go to shared memory by list entry; a thread a cell and field adds them in list
//    order, finds the neighbours' extrema by integer comparison and limits;
//  * the AREPO limiter's minimum over faces of (phi_ext - phi)/dphi is reached at the
//    largest |dphi| of either sign, the numerator being common and rounding monotonic: two
//    quotients a field instead of one a face, and none where it would be at least 1.
//    Which face that is is settled in FP32 (gradient_changes), and its dphi alone formed in
//    FP64: a step of 256 x 256 cells 250 -> 240 us, of 1024 x 1024 3.32 -> 3.21 ms.  (The
//    products with the area by 64-bit integers, eight FP64 instructions a face fewer, measured
//    no faster: 3.23 ms.)
// A block that meets anything unusual -- an index out of range, a cell that its face does not
// name, more list entries than the shared arrays hold, an operand outside the seeds' windows
// -- does its rows on the plain path, status bits included.  Measured at 160,000 cells: 828 ->
// 162 us, 1971 -> 104 FP64 instructions a warp (of 32 rows before, of 8 now), 70% of the pipe.
template <int NC>
struct GradShared {
    static constexpr int CAP = 8 * NC;              // list entries: six a cell on average
    double q[8][CAP], sep[2][CAP], pj[4][CAP];
    double cx[2][NC];                               // the rows' centroids x + dcom
    float sepf[2][CAP];                             // sep over about the cell's size
    int esc[NC];                                    // the exponent of that size
    int fid[CAP], other[CAP];
    unsigned char slot[CAP];
    int task[2][CAP];                               // two-sided from the front, one-sided
    int cell[NC], c[NC], off[NC + 1], ptr[NC], nreal[NC];
    int ntask[2], odd;
    double res_v[4][NC];                            // TESS: each field's minimum, and where
    int res_e[4][NC];
};

// The entry of the block's row t whose face is fid (its first), or -1.
template <int NC>
__device__ __forceinline__ int find_entry(const GradShared<NC> &S, int t, int fid) {
    for (int k = S.off[t]; k < S.off[t + 1]; k++)
        if (S.fid[k] == fid) return k;
    return -1;
}

// The separation of entry k's face from its row's centroid.
template <int NC>
__device__ __forceinline__ void gradient_sep(GradShared<NC> &S, int k, double comx, double comy) {
    const int s = S.slot[k], e = S.esc[s];
    const double sx = comx - S.cx[0][s], sy = comy - S.cx[1][s];
    S.sep[0][k] = sx;
    S.sep[1][k] = sy;
    S.sepf[0][k] = f64_to_f32_scaled(sx, e);
    S.sepf[1][k] = f64_to_f32_scaled(sy, e);
}

// The largest and the smallest change gx sep_x + gy sep_y over the entries k0 .. k1 - 1 (at
// least and at most 0), and the first entries that reach them (-1: none does).  The entry
// is found in FP32: both factors scaled to about 1 and truncated, a change is off by less
// than 2^-21 of M = max(|gx sep_x| + |gy sep_y|), so an entry whose FP32 value leads all others by
// more than 2^-19 M is the one, and its change alone is formed in FP64; otherwise (ties,
// magnitudes beyond the scaling) all are.
template <int NC>
__device__ __forceinline__ void gradient_changes(const GradShared<NC> &S, int k0, int k1, int s, double gx, double gy,
                                                 double &hi, double &lo, int &ehi, int &elo) {
    hi = lo = 0.;
    ehi = elo = -1;
    if ((f64_zero(gx) && f64_zero(gy)) || k0 >= k1) return;
    const unsigned ax = f64_hi(gx) & 0x7fffffffu, ay = f64_hi(gy) & 0x7fffffffu;
    const int e = (int)((ax > ay ? ax : ay) >> 20) - 1023;
    const float fx = f64_to_f32_scaled(gx, e), fy = f64_to_f32_scaled(gy, e);
    float h1 = -INFINITY, h2 = -INFINITY, l1 = INFINITY, l2 = INFINITY, m = 0.f;
    int kh = k0, kl = k0;
    bool bad = e < -890;
    for (int k = k0; k < k1; k++) {
        const float px = fx * S.sepf[0][k], py = fy * S.sepf[1][k], a = px + py;
        m = fmaxf(m, fabsf(px) + fabsf(py));
        bad = bad || !(fabsf(a) < INFINITY);
        h2 = fmaxf(h2, fminf(a, h1));
        l2 = fminf(l2, fmaxf(a, l1));
        if (a > h1) { h1 = a; kh = k; }
        if (a < l1) { l1 = a; kl = k; }
    }
    const float tol = 1.9073486328125e-6f * m;
    if (!bad && m > 8.271806e-25f && h1 - h2 > tol && l2 - l1 > tol) {
        const double dh = gx * S.sep[0][kh] + gy * S.sep[1][kh], dl = gx * S.sep[0][kl] + gy * S.sep[1][kl];
        if (f64_pos(dh)) { hi = dh; ehi = kh; }
        if (f64_neg(dl)) { lo = dl; elo = kl; }
        return;
    }
    for (int k = k0; k < k1; k++) {
        const double dphi = gx * S.sep[0][k] + gy * S.sep[1][k];
        if (f64_lt(hi, dphi)) { hi = dphi; ehi = k; }
        if (f64_lt(dphi, lo)) { lo = dphi; elo = k; }
    }
}

template <int NC, bool TAPE>
__global__ void __launch_bounds__(4 * NC, 5) k_gradients(const __grid_constant__ phd_mesh M, const double *prim, int limiter,
                                                      double *__restrict__ grad, phd_clock *clk, GradTape tape,
                                                      double *__restrict__ w, double gamma, double eta, int regularize) {
    __shared__ GradShared<NC> S;
    const int n = M.n_cells, F = M.n_faces, tid = threadIdx.x, c0 = blockIdx.x * NC;
    if (tid == 0) { S.ntask[0] = S.ntask[1] = 0; S.odd = 0; }
    // rows, their source cells and list bounds
    if (tid < NC) {
        const int i = c0 + tid;
        int c = -1, real = 0, e0 = 0, len = 0;
        if (i < n) {
            real = M.tag[i] == PHD_REAL_TAG;
            c = real ? i : M.map[i];
            if (c < 0 || c >= n) c = -1;
            else {
                e0 = M.nbr_ptr[c];
                len = M.nbr_ptr[c + 1] - e0;
            }
        }
        S.c[tid] = c;
        S.nreal[tid] = real;
        S.ptr[tid] = e0;
        S.cell[tid] = len;
    }
    __syncthreads();
    static_assert(4 * NC >= 32 + NC, "the second warp holds a thread a row");
    if (tid >= 32 && tid < 32 + NC) {
        const int s = tid - 32, c = S.c[s];
        if (c >= 0) {
            S.cx[0][s] = M.x[c] + M.dcom[c];
            S.cx[1][s] = M.x[(size_t)n + c] + M.dcom[(size_t)n + c];
            S.esc[s] = ((int)((f64_hi(M.vol[c]) >> 20) & 0x7ffu) - 1023) >> 1;
        }
    }
    if (tid < 32) {                                  // exclusive scan of the lengths
        int run = 0;
#pragma unroll
        for (int b = 0; b < NC; b += 32) {
            const int len = b + tid < NC ? S.cell[b + tid] : 0;
            int inc = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, inc, o);
                if (tid >= o) inc += t;
            }
            if (b + tid < NC) S.off[b + tid] = run + inc - len;
            if (len < 0) S.odd = 1;
            run += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (tid == 0) {
            S.off[NC] = run;
            if (run > GradShared<NC>::CAP) S.odd = 1;
        }
    }
    __syncthreads();
    const int E = S.off[NC];
    bool ok = true;
    if (!S.odd) {
        for (int k = tid; k < E; k += 4 * NC) {
            int lo = 0, hi = NC;                     // off[lo] <= k < off[hi]
#pragma unroll
            for (int s = NC; s > 1; s >>= 1) {
                const int mid = (lo + hi) >> 1;
                if (S.off[mid] <= k) lo = mid;
                else hi = mid;
            }
            S.slot[k] = (unsigned char)lo;
            S.fid[k] = M.nbr_idx[S.ptr[lo] + (k - S.off[lo])];
        }
    }
    __syncthreads();
    if (!S.odd) {
        for (int k = tid; k < E; k += 4 * NC) {
            const int s = S.slot[k], c = S.c[s], fid = S.fid[k];
            int a = -1, b = -1;
            if (fid >= 0 && fid < F) {
                a = M.pair_i[fid];
                b = M.pair_j[fid];
            }
            const int j = (c == a) ? b : a;
            if ((c != a && c != b) || j < 0 || j >= n) { ok = false; continue; }
            S.other[k] = j;
            const int t = j - c0;                    // the other cell's row, when it is in this block
            int k2 = -1;
            if (j != c && t >= 0 && t < NC && S.nreal[t] && S.nreal[s]) k2 = find_entry(S, t, fid);
            if (k2 >= 0) {
                if (c == a) S.task[0][atomicAdd(&S.ntask[0], 1)] = k | (k2 << 16);
                else if (find_entry(S, s, fid) != k) ok = false;        // the same face twice in a list
            } else {
                S.task[1][atomicAdd(&S.ntask[1], 1)] = k;
            }
        }
        if (!ok) S.odd = 1;
    }
    pdl_wait();                                      // prim: the previous step's update
    // a moving step's generator velocities, each row's own
    if (w && tid >= 3 * NC && c0 + tid - 3 * NC < n)
        generator_velocity(M, prim, gamma, eta, regularize, c0 + tid - 3 * NC, w);
    __syncthreads();
    if (!S.odd) {
        const int n2 = S.ntask[0], nt = n2 + S.ntask[1];
        for (int t = tid; t < nt; t += 4 * NC) {
            const int code = t < n2 ? S.task[0][t] : S.task[1][t - n2];
            const bool two = t < n2;
            const int k = code & 0xffff, k2 = code >> 16;
            const int c = S.c[S.slot[k]], j = S.other[k], fid = S.fid[k];
            const double xc = M.x[c], yc = M.x[(size_t)n + c], xj = M.x[j], yj = M.x[(size_t)n + j];
            const double comx = M.com[fid], comy = M.com[(size_t)F + fid], area = M.area[fid];
            const double cfx = fma(-0.5, xc + xj, comx), cfy = fma(-0.5, yc + yj, comy);
            const double drx = xc - xj, dry = yc - yj;
            const double r = f64_sqrt(drx * drx + dry * dry, ok);
            const double rc = r * M.vol[c], rj = two ? r * M.vol[j] : 1.0;
            const double ic = f64_rcp(rc, ok), ij = f64_rcp(rj, ok);
            gradient_sep(S, k, comx, comy);
            if (two) gradient_sep(S, k2, comx, comy);
#pragma unroll
            for (int f = 0; f < 4; f++) {
                const double pc = prim[(size_t)f * n + c], pj = prim[(size_t)f * n + j];
                const double d_dif = pj - pc, d_sum = pj + pc;
                const double nx = area * fma(-0.5, d_sum * drx, d_dif * cfx);
                const double ny = area * fma(-0.5, d_sum * dry, d_dif * cfy);
                S.q[2 * f][k] = f64_div_by(nx, rc, ic, ok);
                S.q[2 * f + 1][k] = f64_div_by(ny, rc, ic, ok);
                S.pj[f][k] = pj;
                if (two) {
                    S.q[2 * f][k2] = -f64_div_by(nx, rj, ij, ok);
                    S.q[2 * f + 1][k2] = -f64_div_by(ny, rj, ij, ok);
                    S.pj[f][k2] = pc;
                }
            }
        }
        if (!ok) S.odd = 1;
    }
    __syncthreads();
    const int s = tid % NC, f = tid / NC, i = c0 + s;
    const int c = S.c[s];
    double gx = 0., gy = 0., alpha = 1.0;
    int act = -1, emax = -1, emin = -1;
    if (!S.odd && c >= 0) {
        const double pc = prim[(size_t)f * n + c];
        const int k0 = S.off[s], k1 = S.off[s + 1];
        double pmax = pc, pmin = pc;
        long long kmax = f64_key(pc), kmin = kmax;
        for (int k = k0; k < k1; k++) {
            gx = gx + S.q[2 * f][k];
            gy = gy + S.q[2 * f + 1][k];
            const double pj = S.pj[f][k];
            const long long kp = f64_key(pj);
            if (kp > kmax) { kmax = kp; pmax = pj; emax = k; }
            if (kp < kmin) { kmin = kp; pmin = pj; emin = k; }
        }
        if (limiter == PHD_LIMITER_AREPO) {
            double hi, lo;
            int ehi, elo;
            gradient_changes(S, k0, k1, s, gx, gy, hi, lo, ehi, elo);
            const double up = pmax - pc, dn = pmin - pc;
            double ph = 1.0, pl = 1.0;
            if (f64_lt(up, hi)) ph = f64_div(up, hi, ok);
            if (f64_lt(lo, dn)) pl = f64_div(dn, lo, ok);
            ph = f64_max(ph, 0.);
            pl = f64_max(pl, 0.);
            alpha = f64_min(f64_min(ph, pl), 1.0);
            if (TAPE && f64_lt(alpha, 1.0)) {
                // the first entry in list order that reaches the minimum
                int e = f64_lt(pl, ph) ? elo : ehi;
                if (f64_key(ph) == f64_key(pl)) e = min(ehi, elo);
                act = f64_pos(alpha) ? e : -2;
            }
        } else if (limiter == PHD_LIMITER_TESS) {
            for (int k = k0; k < k1; k++) {
                const double dphi = gx * S.sep[0][k] + gy * S.sep[1][k], num = S.pj[f][k] - pc;
                if (f64_zero(dphi)) continue;                            // psi = 1
                double psi = 0.;                                         // opposite signs, or a flat neighbour
                if (!f64_zero(num) && (f64_bits(num) ^ f64_bits(dphi)) >= 0) {
                    const long long m = 0x7fffffffffffffffll;
                    if ((f64_bits(num) & m) >= (f64_bits(dphi) & m)) continue;       // psi >= 1
                    psi = f64_div(num, dphi, ok);
                }
                if (f64_lt(psi, alpha)) { alpha = psi; act = k; }
            }
            S.res_v[f][s] = alpha;
            S.res_e[f][s] = act;
        }
        if (!ok) S.odd = 1;
    }
    __syncthreads();
    if (S.odd) {                                     // uniform over the block
        if (tid < NC && i < n) {
            if (c < 0) set_status(clk, PHD_STATUS_BAD_INDEX);
            else set_status(clk, gradient_row_plain<TAPE>(&M, prim, limiter, i, c, grad, tape));
        }
        return;
    }
    if (i >= n) return;
    if (c < 0) {
        if (f == 0) set_status(clk, PHD_STATUS_BAD_INDEX);
        return;
    }
    int act_f0 = -1;
    if (limiter == PHD_LIMITER_TESS) {
        // every field limits the density's slope alone (reconstruction.pyx:731); the minimum
        // over faces and fields, the first in that order
        alpha = 1.0;
        act = -1;
        if (f == 0) {
            int e = -1;
#pragma unroll
            for (int g = 0; g < 4; g++) {
                const double v = S.res_v[g][s];
                const int ke = S.res_e[g][s];
                if (ke >= 0 && (f64_lt(v, alpha) || (f64_key(v) == f64_key(alpha) && e >= 0 && ke < e))) {
                    alpha = v;
                    e = ke;
                    act_f0 = g;
                }
            }
            if (TAPE) act = e < 0 ? -1 : (f64_pos(alpha) ? e : -2);
        }
    }
    if (TAPE && i == c) {
        const int g0 = S.ptr[s] - S.off[s];          // entry of the block -> list entry
        tape.f64[(size_t)(2 * f) * n + i] = gx;
        tape.f64[(size_t)(2 * f + 1) * n + i] = gy;
        tape.f64[(size_t)(8 + f) * n + i] = alpha;
        tape.i32[(size_t)f * n + i] = act >= 0 ? act + g0 : act;
        tape.i32[(size_t)(4 + f) * n + i] = emax >= 0 ? emax + g0 : -1;
        tape.i32[(size_t)(8 + f) * n + i] = emin >= 0 ? emin + g0 : -1;
        if (f == 0) tape.i32[(size_t)12 * n + i] = act_f0;
    }
    const int fl = M.flip ? M.flip[i] : 0;
    double ox = alpha * gx, oy = alpha * gy;
    if (f == 1 && (fl & 1)) ox = -ox;
    if (f == 2 && (fl & 2)) oy = -oy;
    grad[(size_t)(2 * f) * n + i] = ox;
    grad[(size_t)(2 * f + 1) * n + i] = oy;
}

template <int DIM>
__device__ __forceinline__ void load_face_inputs(const phd_mesh &M, const double *prim,
                                                 const double *grad, const double *face_w,
                                                 int m, int i, int j, bool linear, double *pi, double *pj,
                                                 double *gi, double *gj, double *w) {
    constexpr int NF = DIM + 2;
    const int n = M.n_cells, F = M.n_faces;
#pragma unroll
    for (int f = 0; f < NF; f++) { pi[f] = prim[(size_t)f * n + i]; pj[f] = prim[(size_t)f * n + j]; }
    if (linear) {
#pragma unroll
        for (int r = 0; r < NF * DIM; r++) { gi[r] = grad[(size_t)r * n + i]; gj[r] = grad[(size_t)r * n + j]; }
    }
#pragma unroll
    for (int k = 0; k < DIM; k++) w[k] = face_w ? face_w[(size_t)k * F + m] : 0.0;
}

template <int DIM>
__device__ __forceinline__ void face_states_f64(const phd_mesh &M, int m, int i, int j, const double *pi,
                                                const double *pj, const double *gi, const double *gj,
                                                const double *w, double gamma, double dt_half, bool boost,
                                                bool linear, bool gizmo, double *L, double *R) {
    constexpr int NF = DIM + 2;
    if (linear) {
        face_spatial_f64<DIM>(M, m, i, j, pi, pj, gi, gj, w, boost, gizmo, L, R);
        temporal<double, DIM>(L, R, pi, pj, gi, gj, w, gamma, dt_half, boost);
    } else {                                   // PieceWiseConstant :323-352
#pragma unroll
        for (int f = 0; f < NF; f++) { L[f] = pi[f]; R[f] = pj[f]; }
        if (boost) {
#pragma unroll
            for (int k = 0; k < DIM; k++) { L[1 + k] = pi[1 + k] - w[k]; R[1 + k] = pj[1 + k] - w[k]; }
        }
    }
}

// The face's geometry (linear: with the cells' centroids) and its cell values (linear: with the
// gradients) for the lean states.
__device__ __forceinline__ void load_geometry64(const phd_mesh &M, int m, int i, int j, bool linear, Face64 &A) {
    const int n = M.n_cells, F = M.n_faces;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        A.xi[k] = M.x[(size_t)k * n + i];
        A.xj[k] = M.x[(size_t)k * n + j];
        A.com[k] = M.com[(size_t)k * F + m];
    }
    if (linear) {
#pragma unroll
        for (int k = 0; k < 2; k++) {
            A.ci[k] = M.dcom[(size_t)k * n + i];
            A.cj[k] = M.dcom[(size_t)k * n + j];
        }
    }
}
__device__ __forceinline__ void load_values64(const phd_mesh &M, const double *prim,
                                              const double *grad, int i, int j, bool linear, Face64 &A) {
    const int n = M.n_cells;
#pragma unroll
    for (int f = 0; f < 4; f++) { A.pi[f] = prim[(size_t)f * n + i]; A.pj[f] = prim[(size_t)f * n + j]; }
    if (linear) {
#pragma unroll
        for (int r = 0; r < 8; r++) { A.gi[r] = grad[(size_t)r * n + i]; A.gj[r] = grad[(size_t)r * n + j]; }
    }
}

// One face's states on the plain path: both stages, or the one asked for.
__device__ __noinline__ void states_plain(const phd_mesh *M, const double *prim, const double *grad, const double *face_w,
                                          double gamma, double dt_half, int boost, int linear, int gizmo, int stages,
                                          int m, int i, int j, double *left, double *right) {
    const int F = M->n_faces;
    double pi[4], pj[4], gi[8], gj[8], w[2], L[4], R[4];
    load_face_inputs<2>(*M, prim, grad, face_w, m, i, j, linear, pi, pj, gi, gj, w);
    if (!linear || stages == (PHD_STAGE_SPATIAL | PHD_STAGE_TEMPORAL)) {
        face_states_f64<2>(*M, m, i, j, pi, pj, gi, gj, w, gamma, dt_half, boost, linear, gizmo, L, R);
    } else if (stages == PHD_STAGE_SPATIAL) {
        face_spatial_f64<2>(*M, m, i, j, pi, pj, gi, gj, w, boost, gizmo, L, R);
    } else {
#pragma unroll
        for (int f = 0; f < 4; f++) { L[f] = left[(size_t)f * F + m]; R[f] = right[(size_t)f * F + m]; }
        temporal<double, 2>(L, R, pi, pj, gi, gj, w, gamma, dt_half, boost);
    }
#pragma unroll
    for (int f = 0; f < 4; f++) { left[(size_t)f * F + m] = L[f]; right[(size_t)f * F + m] = R[f]; }
}

// compute_states by itself (the plugin's stage): the lean states for the whole stage, the
// plain ones for a single one of its two halves.
__global__ void __launch_bounds__(128) k_states(const __grid_constant__ phd_mesh M, const __grid_constant__ Gas64 C,
                                                const double *__restrict__ prim, const double *__restrict__ grad,
                                                const double *__restrict__ face_w, double dt_half, int boost, int linear,
                                                int gizmo, int stages, double *left, double *right) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M.n_faces) return;
    const int F = M.n_faces, i = M.pair_i[m], j = M.pair_j[m];
    if (i < 0 || i >= M.n_cells || j < 0 || j >= M.n_cells) return;
    bool ok = false;
    if (!linear || stages == (PHD_STAGE_SPATIAL | PHD_STAGE_TEMPORAL)) {
        Face64 A;
        load_geometry64(M, m, i, j, linear, A);
        load_values64(M, prim, grad, i, j, linear, A);
        A.w[0] = face_w ? face_w[m] : 0.0;
        A.w[1] = face_w ? face_w[(size_t)F + m] : 0.0;
        double L[4], R[4];
        ok = states64(A, C, dt_half, boost, linear, gizmo, L, R);
        if (ok) {
#pragma unroll
            for (int f = 0; f < 4; f++) { left[(size_t)f * F + m] = L[f]; right[(size_t)f * F + m] = R[f]; }
        }
    }
    if (!ok)
        states_plain(&M, prim, grad, face_w, C.g, dt_half, boost, linear, gizmo, stages, m, i, j, left, right);
}

// compute_fluxes by itself (the plugin's stage).
template <int SOLVER>
__global__ void __launch_bounds__(128) k_riemann(const __grid_constant__ phd_mesh M, const __grid_constant__ Gas64 C,
                                                 const __grid_constant__ Exact64 X, int boost, int max_iter, const double *__restrict__ left,
                                                 const double *__restrict__ right, const double *__restrict__ face_w,
                                                 double *__restrict__ flux, phd_clock *clk) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M.n_faces) return;
    const int F = M.n_faces;
    double L[4], R[4], nrm[2], w[2], f[4];
    unsigned big = 0;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        L[q] = left[(size_t)q * F + m];
        R[q] = right[(size_t)q * F + m];
        big = f64_magmax(f64_magmax(big, L[q]), R[q]);
    }
#pragma unroll
    for (int k = 0; k < 2; k++) {
        nrm[k] = M.normal[(size_t)k * F + m];
        w[k] = face_w ? face_w[(size_t)k * F + m] : 0.0;
        big = f64_magmax(big, w[k]);
    }
    bool ok = false, failed = false;
    if (big < F64_FACE_MAX && C.ok) {
        if (SOLVER == PHD_EXACT) ok = exact64_flux(L, R, nrm, w, X, max_iter, f, &failed);
        else ok = hll64<SOLVER == PHD_HLLC>(L, R, nrm, w, C, boost != 0, f);
    }
    if (!ok) failed = false;
    if (!ok) riemann_flux<double, 2>(SOLVER, L, R, nrm, w, C.g, boost != 0, max_iter, f, &failed);
    if (failed) set_status(clk, PHD_STATUS_RIEMANN_NONCONVERGED);
#pragma unroll
    for (int q = 0; q < 4; q++) flux[(size_t)q * F + m] = f[q];
}

// assign_face_velocities mesh.pyx:462-477 for one face from its cells' generator velocities.
__device__ __forceinline__ void face_velocity_plain(const phd_mesh &M, int m, int i, int j, const double *wi,
                                                    const double *wj, double *fw) {
    const int n = M.n_cells, F = M.n_faces;
    double factor = 0.0, denom = 0.0;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const double xi = M.x[(size_t)k * n + i], xj = M.x[(size_t)k * n + j];
        factor = factor + ((wi[k] - wj[k]) * (M.com[(size_t)k * F + m] - (0.5 * (xi + xj))));
        denom = denom + t_sq(xj - xi);
    }
    factor = factor / denom;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const double xi = M.x[(size_t)k * n + i], xj = M.x[(size_t)k * n + j];
        fw[k] = (0.5 * (wi[k] + wj[k])) + (factor * (xj - xi));
    }
}

// One face on the plain path; returns status bits.  w (moving): the generator velocities.
__device__ __noinline__ int face_flux_plain(const phd_mesh *M, const phd_params *P, const double *prim,
                                            const double *grad, const double *w, double *face_w, double dt_half,
                                            int m, int i, int j, double *flux) {
    const int n = M->n_cells, F = M->n_faces;
    const bool boost = (P->solver == PHD_EXACT) ? true : (P->boost != 0);
    const bool linear = P->reconstruction == PHD_LINEAR;
    double pi[4], pj[4], gi[8], gj[8], fw[2], L[4], R[4], nrm[2], f[4];
    if (w) {
        const double wi[2] = {w[i], w[(size_t)n + i]}, wj[2] = {w[j], w[(size_t)n + j]};
        face_velocity_plain(*M, m, i, j, wi, wj, fw);
        face_w[m] = fw[0];
        face_w[(size_t)F + m] = fw[1];
    }
    load_face_inputs<2>(*M, prim, grad, face_w, m, i, j, linear, pi, pj, gi, gj, fw);
    face_states_f64<2>(*M, m, i, j, pi, pj, gi, gj, fw, P->gamma, dt_half, boost, linear, P->gizmo != 0, L, R);
#pragma unroll
    for (int k = 0; k < 2; k++) nrm[k] = M->normal[(size_t)k * F + m];
    bool failed = false;
    riemann_flux<double, 2>(P->solver, L, R, nrm, fw, P->gamma, boost, P->exact_max_iter, f, &failed);
#pragma unroll
    for (int q = 0; q < 4; q++) flux[(size_t)q * F + m] = f[q];
    return failed ? PHD_STATUS_RIEMANN_NONCONVERGED : 0;
}

// Fused: (moving) face velocity, states, Riemann flux and deboost per face; the states never
// reach memory.  Bound by the FP64 pipe: see phd_face64.cuh for how the same numbers come
// out of a third of the FP64 instructions.  The plain path stands in for a face with
// unusual operands.  128 threads at 128 registers: 16 warps a SM, four times what keeps the
// FP64 pipe fed.  Measured (160,000 cells, shear layer, HLLC): 1032 us and 35 us for the face
// velocities by themselves -> 291 us, 1106 + 33 -> 295 FP64 instructions per warp.
template <int SOLVER>
__global__ void __launch_bounds__(128) k_face_flux(const __grid_constant__ phd_mesh M, const __grid_constant__ phd_params P,
                                                   const __grid_constant__ Gas64 C, const __grid_constant__ Exact64 X,
                                                   const double *prim,
                                                   const double *grad, const double *w,
                                                   double *__restrict__ face_w, double *__restrict__ flux,
                                                   phd_clock *clk) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = M.n_cells, F = M.n_faces;
    if (m >= F) return;
    const int i = M.pair_i[m], j = M.pair_j[m];
    if (i < 0 || i >= n || j < 0 || j >= n) {
        pdl_wait();                                  // no kernel is done before the ones ahead of it
        set_status(clk, PHD_STATUS_BAD_INDEX);
        return;
    }
    const bool boost = SOLVER == PHD_EXACT || P.boost != 0;
    const bool linear = P.reconstruction == PHD_LINEAR;
    Face64 A;
    load_geometry64(M, m, i, j, linear, A);
    pdl_wait();                                      // prim, grad, w, the clock: earlier kernels'
    const double dt_half = 0.5 * clk->dt;
    load_values64(M, prim, grad, i, j, linear, A);
    bool ok = true;
    if (w) {
        const double wi[2] = {w[i], w[(size_t)n + i]}, wj[2] = {w[j], w[(size_t)n + j]};
        const double dx = A.xj[0] - A.xi[0], dy = A.xj[1] - A.xi[1];
        const double num = (wi[0] - wj[0]) * fma(-0.5, A.xi[0] + A.xj[0], A.com[0]) +
                           (wi[1] - wj[1]) * fma(-0.5, A.xi[1] + A.xj[1], A.com[1]);
        const double fac = f64_div(num, dx * dx + dy * dy, ok);
        A.w[0] = fma(0.5, wi[0] + wj[0], fac * dx);
        A.w[1] = fma(0.5, wi[1] + wj[1], fac * dy);
    } else {
        A.w[0] = face_w ? face_w[m] : 0.0;
        A.w[1] = face_w ? face_w[(size_t)F + m] : 0.0;
    }
    const double nrm[2] = {M.normal[m], M.normal[(size_t)F + m]};
    double L[4], R[4], f[4];
    ok = states64(A, C, dt_half, boost, linear, P.gizmo != 0, L, R) && ok;
    int status = 0;
    if (SOLVER == PHD_EXACT) {
        bool failed = false;
        ok = ok && exact64_flux(L, R, nrm, A.w, X, P.exact_max_iter, f, &failed);
        if (failed) status = PHD_STATUS_RIEMANN_NONCONVERGED;
    } else {
        ok = hll64<SOLVER == PHD_HLLC>(L, R, nrm, A.w, C, boost, f) && ok;
    }
    pdl_launch_dependents();                         // 5% of a step with the exact solver's long last warps
    if (ok) {
        if (w) {
            face_w[m] = A.w[0];
            face_w[(size_t)F + m] = A.w[1];
        }
#pragma unroll
        for (int q = 0; q < 4; q++) flux[(size_t)q * F + m] = f[q];
    } else {
        status = face_flux_plain(&M, &P, prim, grad, w, face_w, dt_half, m, i, j, flux);
    }
    set_status(clk, status);
}

// ---- conserved update -----------------------------------------------------------
// u <= 0.0 by the bits (false for a NaN)
__device__ __forceinline__ bool f64_le0(double u) {
    const long long b = f64_bits(u);
    return b <= 0 && (b & 0x7fffffffffffffffll) <= 0x7ff0000000000000ll;
}

// Mesh.update_from_fluxes mesh.pyx:519-551 for cell c as a segmented sum over its
// faces in ascending face id (the order in which the reference's face loop reaches
// it): U -= dt*a*F where c is pair-i, U += dt*a*F where c is pair-j.
template <int DIM>
__device__ __forceinline__ int cell_update_f64(const phd_mesh &M, const double *__restrict__ flux, double dt,
                                               int c, double *U) {
    constexpr int NF = DIM + 2;
    const int F = M.n_faces;
    int status = 0;
    const int m0 = M.nbr_ptr[c], m1 = M.nbr_ptr[c + 1];
    for (int m = m0; m < m1; m++) {
        const int fid = M.nbr_idx[m];
        if (fid < 0 || fid >= F) { status |= PHD_STATUS_BAD_INDEX; continue; }
        const double a = M.area[fid];
        if (M.pair_i[fid] == c) {
#pragma unroll
            for (int q = 0; q < NF; q++) U[q] = U[q] - ((dt * a) * flux[(size_t)q * F + fid]);
        } else {
#pragma unroll
            for (int q = 0; q < NF; q++) U[q] = U[q] + ((dt * a) * flux[(size_t)q * F + fid]);
        }
        if (f64_le0(U[0])) status |= PHD_STATUS_NEG_MASS;
        if (f64_le0(U[DIM + 1])) status |= PHD_STATUS_NEG_ENERGY;
    }
    return status;
}

template <int DIM>
__global__ void __launch_bounds__(BLOCK) k_update(phd_mesh M, const double *__restrict__ flux, double dt,
                                                   double *__restrict__ cons, phd_clock *clk) {
    constexpr int NF = DIM + 2;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= M.n_cells || M.tag[i] != PHD_REAL_TAG) return;
    const int n = M.n_cells;
    double U[NF];
#pragma unroll
    for (int q = 0; q < NF; q++) U[q] = cons[(size_t)q * n + i];
    const int st = cell_update_f64<DIM>(M, flux, dt, i, U);
    set_status(clk, st);
#pragma unroll
    for (int q = 0; q < NF; q++) cons[(size_t)q * n + i] = U[q];
}

template <int DIM>
__global__ void __launch_bounds__(BLOCK) k_ghost_cons(phd_mesh M, double *__restrict__ cons) {
    constexpr int NF = DIM + 2;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= M.n_cells || M.tag[i] == PHD_REAL_TAG) return;
    const int n = M.n_cells, c = M.map[i];
    if (c < 0 || c >= n) return;
    const int fl = M.flip ? M.flip[i] : 0;
#pragma unroll
    for (int q = 0; q < NF; q++) {
        double u = cons[(size_t)q * n + c];
        if (q >= 1 && q <= DIM && (fl & (1 << (q - 1)))) u *= -1;
        cons[(size_t)q * n + i] = u;
    }
}

// IdealGas.primitive_from_conservative equation_state.pyx:106-117 for one cell.
template <int DIM>
__device__ __forceinline__ void prim_of(const double *U, double vol, double gamma, double *p) {
    const double m = U[0];
    const double d = m / vol;
    p[0] = d;
    double v_sq = 0.;
#pragma unroll
    for (int k = 0; k < DIM; k++) {
        const double v = U[1 + k] / m;
        p[1 + k] = v;
        v_sq = v_sq + v * v;
    }
    p[DIM + 1] = ((U[DIM + 1] / vol) - ((.5 * d) * v_sq)) * (gamma - 1.);
}

// CFL candidate of one real cell, RiemannBase.compute_time_step riemann.pyx:170-187.
template <int DIM>
__device__ __forceinline__ double cfl_candidate(const double *p, double vol, double gamma, bool boost) {
    const double c = sqrt((gamma * p[DIM + 1]) / p[0]);
    const double R = (DIM == 2) ? sqrt(vol / 3.141592653589793)
                                : pow((3.0 * vol) / (4.0 * 3.141592653589793), 1.0 / 3.0);
    if (boost) return R / c;
    double vsq = 0.0;
#pragma unroll
    for (int k = 0; k < DIM; k++) vsq = vsq + p[1 + k] * p[1 + k];
    return R / (c + sqrt(vsq));
}

// The recovery of one cell (prim_of) with the quotients of each denominator sharing its seed.
__device__ __forceinline__ void prim_lean(const double *U, double vol, double gamma, double *p) {
    bool ok = true;
    const double ym = f64_rcp(U[0], ok), yv = f64_rcp(vol, ok);
    const double d = f64_div_by(U[0], vol, yv, ok);
    const double vx = f64_div_by(U[1], U[0], ym, ok), vy = f64_div_by(U[2], U[0], ym, ok);
    p[0] = d;
    p[1] = vx;
    p[2] = vy;
    p[3] = fma(-0.5, d * (vx * vx + vy * vy), f64_div_by(U[3], vol, yv, ok)) * (gamma - 1.);
    if (!ok) prim_of<2>(U, vol, gamma, p);
}

// The CFL candidate (cfl_candidate) with seeded quotients and roots.
__device__ __forceinline__ double cfl_lean(const double *p, double vol, double gamma, bool boost) {
    bool ok = true;
    const double c = f64_sqrt(f64_div(gamma * p[3], p[0], ok), ok);
    const double R = f64_sqrt(f64_div_by(vol, 3.141592653589793, 1.0 / 3.141592653589793, ok), ok);
    double den = c;
    if (!boost) {
        const double vsq = p[1] * p[1] + p[2] * p[2];
        den = c + (f64_zero(vsq) ? 0. : f64_sqrt(vsq, ok));
    }
    const double cand = f64_div(R, den, ok);
    return ok ? cand : cfl_candidate<2>(p, vol, gamma, boost);
}

__global__ void __launch_bounds__(BLOCK) k_prim_from_cons(int n, double gamma, const double *__restrict__ vol,
                                                           const double *__restrict__ cons, double *__restrict__ prim) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double U[4], p[4];
#pragma unroll
    for (int q = 0; q < 4; q++) U[q] = cons[(size_t)q * n + i];
    prim_lean(U, vol[i], gamma, p);
#pragma unroll
    for (int q = 0; q < 4; q++) prim[(size_t)q * n + i] = p[q];
}

// IdealGas.conservative_from_primitive equation_state.pyx:65-79.
template <int DIM>
__global__ void __launch_bounds__(BLOCK) k_cons_from_prim(int n, double gamma, const double *__restrict__ vol,
                                                           const double *__restrict__ prim, double *__restrict__ cons) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double d = prim[i];
    const double m = d * vol[i];
    cons[i] = m;
    double v_sq = 0.;
#pragma unroll
    for (int k = 0; k < DIM; k++) {
        const double v = prim[(size_t)(1 + k) * n + i];
        cons[(size_t)(1 + k) * n + i] = v * m;
        v_sq = v_sq + v * v;
    }
    cons[(size_t)(DIM + 1) * n + i] = (((.5 * d) * v_sq) + (prim[(size_t)(DIM + 1) * n + i] / (gamma - 1.))) * vol[i];
}

__global__ void __launch_bounds__(BLOCK) k_time_step(phd_mesh M, const double *__restrict__ prim, double gamma,
                                                      double cfl, int boost, int advance, phd_clock *clk) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = M.n_cells;
    double cand = INFINITY;
    if (i < n && M.tag[i] == PHD_REAL_TAG) {
        double p[4];
#pragma unroll
        for (int q = 0; q < 4; q++) p[q] = prim[(size_t)q * n + i];
        cand = cfl_lean(p, M.vol[i], gamma, boost != 0);
    }
    block_min_to(cand, &clk->dtmin_bits);
    finish_cfl(clk, cfl, advance != 0);
}

// Fused end of step: segmented update into cons_next (ghosts redo their image's sum
// and flip the reflective momentum), primitive recovery for every cell and the CFL
// minimum over real cells for the next step.  The sums are cell_update_f64's, face after face
// in list order; the loads of four faces go out together.  The time-step candidates are
// compared in FP32 first and only the cells within its rounding of the block's smallest
// form theirs in FP64: 16 FP64 instructions fewer in the other warps, 100 left.  (Four threads a
// cell, one a field, measured no faster at 16,000 cells and 99 us against 58 at 160,000: each
// then forms dt A by itself; with dt A handed round, 64.0 -> 63.4 us a step at 10,000 cells but 480 ->
// 504 for two at 66,000.)  Measured at 160,000 cells: 90.6 -> 48.0 us.
__global__ void __launch_bounds__(128) k_update_step(const __grid_constant__ phd_mesh M,
                                                     const __grid_constant__ phd_params P,
                                                     const double *flux, const double *cons,
                                                     double *__restrict__ cons_next, double *__restrict__ prim,
                                                     phd_clock *clk) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = M.n_cells, F = M.n_faces;
    const bool boost = (P.solver == PHD_EXACT) ? true : (P.boost != 0);
    double p[4] = {0., 0., 0., 0.}, vol = 0.;
    float c32 = INFINITY;                            // the candidate in FP32; -1: to be formed in any case
    // the row, its list and the first chunk's faces: the mesh's, loaded ahead of the wait
    constexpr int CH = 4;
    int c = -1, m0 = 0, m1 = 0, status = 0, fid[CH], a[CH];
    double ar[CH];
    bool real = false;
    const auto load_faces = [&](int mb) {
#pragma unroll
        for (int k = 0; k < CH; k++) {
            fid[k] = M.nbr_idx[mb + k < m1 ? mb + k : m0];
            if (fid[k] < 0 || fid[k] >= F) fid[k] = -1;
        }
#pragma unroll
        for (int k = 0; k < CH; k++) {
            const int f = fid[k] < 0 ? 0 : fid[k];
            a[k] = M.pair_i[f];
            ar[k] = M.area[f];
        }
    };
    if (i < n) {
        real = M.tag[i] == PHD_REAL_TAG;
        c = real ? i : M.map[i];
        if (c >= 0 && c < n) {
            m0 = M.nbr_ptr[c];
            m1 = M.nbr_ptr[c + 1];
            vol = M.vol[i];
            if (F <= 0 && m1 > m0) { status |= PHD_STATUS_BAD_INDEX; m1 = m0; }
            if (m0 < m1) load_faces(m0);
        } else {
            c = -1;
            status |= PHD_STATUS_BAD_INDEX;
        }
    }
    pdl_wait();                                      // flux: the face kernel's; cons, the clock
    if (c >= 0) {
        const double dt = clk->dt;
        double U[4];
#pragma unroll
        for (int q = 0; q < 4; q++) U[q] = cons[(size_t)q * n + c];
        for (int mb = m0; mb < m1; mb += CH) {
            if (mb != m0) load_faces(mb);
            double fl[CH][4];
#pragma unroll
            for (int k = 0; k < CH; k++)
#pragma unroll
                for (int q = 0; q < 4; q++) fl[k][q] = flux[(size_t)q * F + (fid[k] < 0 ? 0 : fid[k])];
#pragma unroll
            for (int k = 0; k < CH; k++) {
                if (mb + k >= m1) break;
                if (fid[k] < 0) { status |= PHD_STATUS_BAD_INDEX; continue; }
                const double da = dt * ar[k];
                const long long sg = a[k] == c ? (long long)0x8000000000000000ull : 0ll;
#pragma unroll
                for (int q = 0; q < 4; q++) U[q] = U[q] + f64_from(f64_bits(da * fl[k][q]) ^ sg);
                if (f64_le0(U[0])) status |= PHD_STATUS_NEG_MASS;
                if (f64_le0(U[3])) status |= PHD_STATUS_NEG_ENERGY;
            }
        }
        if (!real) {
            const int fl = M.flip ? M.flip[i] : 0;
            if (fl & 1) U[1] = -U[1];
            if (fl & 2) U[2] = -U[2];
        }
        prim_lean(U, vol, P.gamma, p);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            cons_next[(size_t)q * n + i] = U[q];
            prim[(size_t)q * n + i] = p[q];
        }
        if (real) {
            // R/c within a few FP32 roundings while the operands and p/rho are well inside FP32's
            // range (where the quotient is subnormal its rounding could hide the smallest)
            const unsigned lo = (1023u - 100u) << 20, span = 200u << 20;
            const float c2 = (float)P.gamma * f64_to_f32(p[3]) / f64_to_f32(p[0]);
            const bool in = f64_hi(p[0]) - lo < span && f64_hi(p[3]) - lo < span && f64_hi(vol) - lo < span &&
                            c2 >= 7.8886091e-31f;
            const float cs = sqrtf(c2);
            const float vx = f64_to_f32(p[1]), vy = f64_to_f32(p[2]);
            const float den = boost ? cs : cs + sqrtf(vx * vx + vy * vy);
            c32 = in ? sqrtf(f64_to_f32(vol) * 0.3183098861837907f) / den : -1.f;
            if (!(c32 < INFINITY && c32 > 0.f)) c32 = -1.f;
        }
    }
    set_status(clk, status);
    __shared__ float s_c32[4];
    const float wmin = warp_min_f(c32 < 0.f ? INFINITY : c32);
    if ((threadIdx.x & 31) == 0) s_c32[threadIdx.x >> 5] = wmin;
    __syncthreads();
    float bmin = s_c32[0];
    for (int k = 1; k < (int)(blockDim.x >> 5); k++) bmin = fminf(bmin, s_c32[k]);
    double cand = INFINITY;
    if (c32 < 0.f || (c32 < INFINITY && c32 <= bmin * (1.f + 1e-5f))) cand = cfl_lean(p, vol, P.gamma, boost);
    block_min_to(cand, &clk->dtmin_bits);
    finish_cfl(clk, P.cfl, true);
}

// ---- mesh motion ------------------------------------------------------------------
// Mesh.assign_generator_velocities mesh.pyx:397-426 (all cells), by itself: the plugin's stage,
// and the steps without gradients.
__global__ void __launch_bounds__(BLOCK) k_gen_vel(const __grid_constant__ phd_mesh M, const double *prim,
                                                   double gamma, double eta, int regularize, double *__restrict__ w) {
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < M.n_cells) generator_velocity(M, prim, gamma, eta, regularize, i, w);
}

// Mesh.assign_face_velocities mesh.pyx:462-477.
template <int DIM>
__global__ void __launch_bounds__(BLOCK) k_face_vel(phd_mesh M, const double *__restrict__ w,
                                                     double *__restrict__ face_w) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M.n_faces) return;
    const int n = M.n_cells, F = M.n_faces;
    const int i = M.pair_i[m], j = M.pair_j[m];
    if (i < 0 || i >= n || j < 0 || j >= n) return;
    const double wi[2] = {w[i], w[(size_t)n + i]}, wj[2] = {w[j], w[(size_t)n + j]};
    double fw[2];
    face_velocity_plain(M, m, i, j, wi, wj, fw);
    face_w[m] = fw[0];
    face_w[(size_t)F + m] = fw[1];
}

inline int blk_of(int n) { return block_for(n, BLOCK); }
inline int grid_of(int n) { return grid_for_block(n, blk_of(n)); }

// Gradients of n rows: blocks of 32 rows and 96 registers, 20 warps an SM (against blocks of 16
// rows at 112 registers, 18 warps: a step of 1024 x 1024 cells 3.19 -> 3.04 ms, of 333 x 333 382 ->
// 356 us; equal below 20,000 cells); w: with a moving step's generator velocities (par's eta
// and regularize).
inline void launch_gradients(const phd_mesh &M, const double *prim, int limiter, double *grad, phd_clock *clk,
                             GradTape tape, double *w, const phd_params *par, PdlQueue &queue) {
    constexpr int NC = 32;
    const int grid = (M.n_cells + NC - 1) / NC;
    const double gamma = par ? par->gamma : 0., eta = par ? par->eta : 0.;
    const int reg = par ? par->regularize : 0;
    if (tape.f64)
        launch_pdl(k_gradients<NC, true>, grid, 4 * NC, queue, M, prim, limiter, grad, clk, tape, w, gamma, eta, reg);
    else
        launch_pdl(k_gradients<NC, false>, grid, 4 * NC, queue, M, prim, limiter, grad, clk, tape, w, gamma, eta, reg);
}

inline void launch_gen_vel(const phd_mesh &M, const double *prim, double gamma, double eta, int regularize, double *w,
                           PdlQueue &queue) {
    const int block = block_for(M.n_cells, BLOCK);
    launch_pdl(k_gen_vel, grid_for_block(M.n_cells, block), block, queue, M, prim, gamma, eta, regularize, w);
}

// Face fluxes; w: the generator velocities of a moving step, from which face_w is formed,
// or null (face_w as given).
inline void launch_face_flux(const phd_mesh &M, const phd_params &P, const double *prim, const double *grad,
                             const double *w, double *face_w, double *flux, phd_clock *clk, PdlQueue &queue) {
    // one warp a block while there are fewer than 16 an SM: the pipe's work is then spread to
    // a warp's grain
    const int block = M.n_faces < 16 * 128 * sm_count_current() ? 32 : 128, grid = grid_for_block(M.n_faces, block);
    const Gas64 C = gas64(P.gamma);
    const Exact64 X = exact64(P.gamma);
    // a number without a name is HLL, as riemann_flux has it
    if (P.solver == PHD_EXACT)
        launch_pdl(k_face_flux<PHD_EXACT>, grid, block, queue, M, P, C, X, prim, grad, w, face_w, flux, clk);
    else if (P.solver == PHD_HLLC)
        launch_pdl(k_face_flux<PHD_HLLC>, grid, block, queue, M, P, C, X, prim, grad, w, face_w, flux, clk);
    else
        launch_pdl(k_face_flux<PHD_HLL>, grid, block, queue, M, P, C, X, prim, grad, w, face_w, flux, clk);
}

inline int launch_status() {
    return cudaPeekAtLastError() == cudaSuccess ? PHD_OK : PHD_ERR_LAUNCH;
}

inline bool mesh_ok(const phd_mesh *M) {
    return M && M->dim == 2 && M->n_cells > 0 && M->n_faces >= 0 && M->n_real <= M->n_cells;
}

}  // namespace phd

using namespace phd;

extern "C" {

int phd_abi_version(void) { return PHDFLUX_ABI_VERSION; }

const char *phd_status_string(int bit) {
    switch (bit) {
        case PHD_STATUS_NEG_MASS: return "Mass less than zero in flux update";
        case PHD_STATUS_NEG_ENERGY: return "Energy less than zero in flux update";
        case PHD_STATUS_RIEMANN_NONCONVERGED: return "No convergence in Exact Riemann Solver";
        case PHD_STATUS_BAD_INDEX: return "ERROR: incorrect neighbors!";
        case PHD_STATUS_LEFT_DOMAIN: return "particle left domain in reflective boundary condition!!";
        case PHD_STATUS_NONFINITE: return "Non-finite primitive state after flux update";
        default: return "unknown status";
    }
}

int phd_gradients_f64(const phd_mesh *mesh, const double *prim, int32_t limiter, double *grad,
                      phd_clock *clk, cudaStream_t stream) {
    if (!mesh_ok(mesh) || !prim || !grad) return PHD_ERR_ARG;
    PdlQueue queue = {stream};
    launch_gradients(*mesh, prim, limiter, grad, clk, GradTape{nullptr, nullptr}, nullptr, nullptr, queue);
    return launch_status();
}

int phd_gradients_f64_taped(const phd_mesh *mesh, const double *prim, int32_t limiter, double *grad,
                            double *tape_f64, int32_t *tape_i32, phd_clock *clk, cudaStream_t stream) {
    if (!mesh_ok(mesh) || !prim || !grad || !tape_f64 || !tape_i32) return PHD_ERR_ARG;
    PdlQueue queue = {stream};
    launch_gradients(*mesh, prim, limiter, grad, clk, GradTape{tape_f64, tape_i32}, nullptr, nullptr, queue);
    return launch_status();
}

int phd_states_f64(const phd_mesh *mesh, const double *prim, const double *grad, const double *face_w,
                   double gamma, double dt_half, int32_t boost, int32_t reconstruction, int32_t gizmo,
                   int32_t stages, double *left, double *right, cudaStream_t stream) {
    if (!mesh_ok(mesh) || !prim || !left || !right) return PHD_ERR_ARG;
    if (reconstruction == PHD_LINEAR && !grad) return PHD_ERR_ARG;
    if (stages < 1 || stages > 3) return PHD_ERR_ARG;
    if (mesh->n_faces == 0) return PHD_OK;
    const int block = block_for(mesh->n_faces, 128);
    k_states<<<grid_for_block(mesh->n_faces, block), block, 0, stream>>>(*mesh, gas64(gamma), prim, grad, face_w, dt_half, boost,
                                                                         reconstruction == PHD_LINEAR, gizmo, stages,
                                                                         left, right);
    return launch_status();
}

int phd_riemann_f64(const phd_mesh *mesh, int32_t solver, double gamma, int32_t boost, int32_t exact_max_iter,
                    const double *left, const double *right, const double *face_w, double *flux,
                    phd_clock *clk, cudaStream_t stream) {
    if (!mesh_ok(mesh) || !left || !right || !flux) return PHD_ERR_ARG;
    if (mesh->n_faces && !mesh->normal) return PHD_ERR_ARG;
    if (solver < PHD_HLL || solver > PHD_EXACT) return PHD_ERR_ARG;
    if (mesh->n_faces == 0) return PHD_OK;
    const int block = block_for(mesh->n_faces, 128), grid = grid_for_block(mesh->n_faces, block);
    const Gas64 C = gas64(gamma);
    const Exact64 X = exact64(gamma);
    if (solver == PHD_HLL)
        k_riemann<PHD_HLL><<<grid, block, 0, stream>>>(*mesh, C, X, boost, exact_max_iter, left, right, face_w, flux, clk);
    else if (solver == PHD_HLLC)
        k_riemann<PHD_HLLC><<<grid, block, 0, stream>>>(*mesh, C, X, boost, exact_max_iter, left, right, face_w, flux, clk);
    else
        k_riemann<PHD_EXACT><<<grid, block, 0, stream>>>(*mesh, C, X, boost, exact_max_iter, left, right, face_w, flux, clk);
    return launch_status();
}

int phd_update_from_fluxes_f64(const phd_mesh *mesh, const double *flux, double dt, double *cons,
                               phd_clock *clk, cudaStream_t stream) {
    if (!mesh_ok(mesh) || !flux || !cons) return PHD_ERR_ARG;
    k_update<2><<<grid_of(mesh->n_cells), blk_of(mesh->n_cells), 0, stream>>>(*mesh, flux, dt, cons, clk);
    return launch_status();
}

int phd_ghost_cons_f64(const phd_mesh *mesh, double *cons, cudaStream_t stream) {
    if (!mesh_ok(mesh) || !cons) return PHD_ERR_ARG;
    k_ghost_cons<2><<<grid_of(mesh->n_cells), blk_of(mesh->n_cells), 0, stream>>>(*mesh, cons);
    return launch_status();
}

int phd_prim_from_cons_f64(int32_t dim, int32_t n, double gamma, const double *vol, const double *cons,
                           double *prim, cudaStream_t stream) {
    if (dim != 2 || n <= 0 || !vol || !cons || !prim) return PHD_ERR_ARG;
    k_prim_from_cons<<<grid_of(n), blk_of(n), 0, stream>>>(n, gamma, vol, cons, prim);
    return launch_status();
}

int phd_cons_from_prim_f64(int32_t dim, int32_t n, double gamma, const double *vol, const double *prim,
                           double *cons, cudaStream_t stream) {
    if (dim != 2 || n <= 0 || !vol || !cons || !prim) return PHD_ERR_ARG;
    k_cons_from_prim<2><<<grid_of(n), blk_of(n), 0, stream>>>(n, gamma, vol, prim, cons);
    return launch_status();
}

int phd_time_step_f64(const phd_mesh *mesh, const double *prim, double gamma, double cfl, int32_t boost,
                      int32_t advance, phd_clock *clk, cudaStream_t stream) {
    if (!mesh_ok(mesh) || !prim || !clk) return PHD_ERR_ARG;
    k_time_step<<<grid_of(mesh->n_cells), blk_of(mesh->n_cells), 0, stream>>>(*mesh, prim, gamma, cfl, boost, advance, clk);
    return launch_status();
}

int phd_generator_velocities_f64(const phd_mesh *mesh, const double *prim, double gamma, double eta,
                                 int32_t regularize, double *w, cudaStream_t stream) {
    if (!mesh_ok(mesh) || !prim || !w) return PHD_ERR_ARG;
    PdlQueue queue = {stream};
    launch_gen_vel(*mesh, prim, gamma, eta, regularize, w, queue);
    return launch_status();
}

int phd_face_velocities_f64(const phd_mesh *mesh, const double *w, double *face_w, cudaStream_t stream) {
    if (!mesh_ok(mesh) || !w || !face_w) return PHD_ERR_ARG;
    if (mesh->n_faces == 0) return PHD_OK;
    k_face_vel<2><<<grid_of(mesh->n_faces), blk_of(mesh->n_faces), 0, stream>>>(*mesh, w, face_w);
    return launch_status();
}

static int step_f64(const phd_mesh *mesh, const phd_params *par, int32_t moving, double *prim, const double *cons,
                    double *cons_next, double *grad, double *w, double *face_w, double *flux, phd_clock *clk,
                    PdlQueue &queue, cudaEvent_t *marks, GradTape tape);

int phd_step_f64_marked(const phd_mesh *mesh, const phd_params *par, int32_t moving, double *prim,
                        const double *cons, double *cons_next, double *grad, double *w, double *face_w,
                        double *flux, phd_clock *clk, cudaStream_t stream, cudaEvent_t *marks) {
    phd::NvtxRange nvtx_range("phd_step_f64");
    PdlQueue queue = {stream};
    return step_f64(mesh, par, moving, prim, cons, cons_next, grad, w, face_w, flux, clk, queue, marks,
                    GradTape{nullptr, nullptr});
}

int phd_step_f64_taped(const phd_mesh *mesh, const phd_params *par, int32_t moving, double *prim,
                       const double *cons, double *cons_next, double *grad, double *w, double *face_w,
                       double *flux, double *tape_f64, int32_t *tape_i32, phd_clock *clk, cudaStream_t stream) {
    phd::NvtxRange nvtx_range("phd_step_f64_taped");
    if (!tape_f64 || !tape_i32) return PHD_ERR_ARG;
    PdlQueue queue = {stream};
    return step_f64(mesh, par, moving, prim, cons, cons_next, grad, w, face_w, flux, clk, queue, nullptr,
                    GradTape{tape_f64, tape_i32});
}

static int step_f64(const phd_mesh *mesh, const phd_params *par, int32_t moving, double *prim, const double *cons,
                    double *cons_next, double *grad, double *w, double *face_w, double *flux, phd_clock *clk,
                    PdlQueue &queue, cudaEvent_t *marks, GradTape tape) {
    if (!mesh_ok(mesh) || !par || !prim || !cons || !cons_next || !flux || !clk) return PHD_ERR_ARG;
    if (mesh->n_faces && !mesh->normal) return PHD_ERR_ARG;
    const bool linear = par->reconstruction == PHD_LINEAR;
    if (linear && !grad) return PHD_ERR_ARG;
    if (moving && (!w || !face_w)) return PHD_ERR_ARG;
    if (marks) cudaEventRecord(marks[0], queue.stream);
    if (linear)
        launch_gradients(*mesh, prim, par->limiter, grad, clk, tape, moving ? w : nullptr, par, queue);
    else if (moving)
        launch_gen_vel(*mesh, prim, par->gamma, par->eta, par->regularize, w, queue);
    if (marks) cudaEventRecord(marks[1], queue.stream);
    if (mesh->n_faces)
        launch_face_flux(*mesh, *par, prim, grad, moving ? w : nullptr, face_w, flux, clk, queue);
    if (marks) cudaEventRecord(marks[2], queue.stream);
    const int bc = block_for(mesh->n_cells, 128);
    launch_pdl(k_update_step, grid_for_block(mesh->n_cells, bc), bc, queue, *mesh, *par, (const double *)flux, cons, cons_next, prim, clk);
    if (marks) cudaEventRecord(marks[3], queue.stream);
    return launch_status();
}

int phd_step_f64(const phd_mesh *mesh, const phd_params *par, int32_t moving, double *prim, const double *cons,
                 double *cons_next, double *grad, double *w, double *face_w, double *flux, phd_clock *clk,
                 cudaStream_t stream) {
    phd::NvtxRange nvtx_range("phd_step_f64");
    return phd_step_f64_marked(mesh, par, moving, prim, cons, cons_next, grad, w, face_w, flux, clk, stream,
                               nullptr);
}

int phd_steps_f64(const phd_mesh *mesh, const phd_params *par, int32_t moving, double *prim, double *cons,
                  double *cons_other, double *grad, double *w, double *face_w, double *flux, phd_clock *clk,
                  int32_t n_steps, cudaStream_t stream) {
    if (n_steps < 0) return PHD_ERR_ARG;
    PdlQueue queue = {stream};
    for (int k = 0; k < n_steps; k++) {
        phd::NvtxRange nvtx_range("phd_step_f64");
        const int rc = step_f64(mesh, par, moving, prim, (k & 1) ? cons_other : cons, (k & 1) ? cons : cons_other, grad, w,
                                face_w, flux, clk, queue, nullptr, GradTape{nullptr, nullptr});
        if (rc != PHD_OK) return rc;
    }
    return PHD_OK;
}

}  // extern "C"
