"""The work this package does for its users, as cases that can be timed and compared.

Each case is one way a program calls the package, at one size: whole steps of a run that
stays on the device (FluxStepper, launched directly or replayed from a CUDA graph), the
hand-over of a new tessellation followed by one step, many small runs advanced together
(EnsembleStepper), the reference's plugin classes called stage by stage, and a
differentiated run forward and backward (FluxRun).  The problems and sizes are the ones
the package is tested and measured on: the reflective shock tube (100 x 100), the point
explosion (256 x 256, periodic), the shear layer (up to 1024 x 1024), the Gaussian bump
(128 x 128) and the two-state ensemble (1,000 to 65,536 cells a run).  A smooth seeded
perturbation is laid over each problem's initial state, so that slopes, limiters and
Riemann fans are at work in every cell, as they are once a run is under way.

exact() restates the scheme in plain torch operations in 64 bits: limited gradients, GIZMO
pair limiter, MUSCL-Hancock half step, HLL / HLLC / exact Riemann flux in the moving face
frame, conserved update, CFL time step.  Its gradients come from torch's autograd.
"""
import importlib
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

pkg = importlib.import_module("phd-code_gb300")
adjoint = importlib.import_module("phd-code_gb300.adjoint")
ensemble = importlib.import_module("phd-code_gb300.ensemble")

F64 = torch.float64
GAMMA = {"tube": 1.4, "explosion": 1.4, "shear": 5.0 / 3.0, "bump": 1.4}


def _case(name, kind, problem, side, steps, precision="fp64", solver="hllc", limiter="arepo",
          reconstruction="linear", boost=True, moving=True, **more):
    c = dict(kind=kind, problem=problem, side=side, steps=steps, precision=precision, solver=solver,
             limiter=limiter, reconstruction=reconstruction, boost=boost, moving=moving, **more)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # a quick look at a small problem: a handful of steps launched one by one, where the
        # launches and the kernels' latency are all there is
        _case("fp32_tube_32", "step", "tube", 32, 8, "fp32", moving=False),
        # the explosion with the exact solver in the fast precision
        _case("fp32_explosion_256_exact", "step", "explosion", 256, 8, "fp32", "exact"),
        # an odd size with the other solver and limiter
        _case("fp32_shear_333_hll_tess", "step", "shear", 333, 8, "fp32", "hll", "tess"),
        # a production run: the largest configuration, replayed from a CUDA graph
        _case("fp32_shear_1024_graph", "graph", "shear", 1024, 10, "fp32"),
        # one step of the moving-mesh loop: a new tessellation from pinned host memory, the
        # step on it, the generator velocities back for the next tessellation
        _case("fp32_remesh_512", "remesh", "shear", 512, 1, "fp32"),
        # many independent small runs, from the smallest to the largest size of the ensemble
        _case("fp32_ensemble_24", "ensemble", "riemann", 256, 4, "fp32", runs=24),
        # the reference's own shock-tube configuration in its own precision, static mesh
        _case("fp64_tube_100", "step", "tube", 100, 8, moving=False),
        # the explosion in the parity precision, HLLC and (at an odd size) the exact solver
        _case("fp64_explosion_256", "step", "explosion", 256, 2),
        _case("fp64_explosion_181_exact", "step", "explosion", 181, 2, solver="exact"),
        # the largest configuration in the parity precision
        _case("fp64_shear_1024", "step", "shear", 1024, 1),
        # the reference's integrator with its plugins on the device, one step with its dt
        _case("fp64_plugins_tube_100", "plugins", "tube", 100, 1),
        # a differentiated run: forward, then backward with recompute from checkpoints
        _case("fp64_adjoint_bump_128", "adjoint", "bump", 128, 40, moving=False, checkpoint=20),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "graph", "remesh", "ensemble", "plugins", "adjoint"])
    solver = rng.choice(["hllc", "hllc", "hll", "exact"])
    limiter = rng.choice(["arepo", "arepo", "arepo", "tess"])
    problem = rng.choice(["tube", "explosion", "shear"])
    moving = rng.random() < 0.6
    if kind == "adjoint":
        return _case(None, kind, "bump", _log_int(rng, 16, 128), rng.randint(3, 40), solver=solver, limiter=limiter,
                     moving=moving, checkpoint=rng.choice([4, 7, 20]))
    if kind == "ensemble":
        return _case(None, kind, "riemann", _log_int(rng, 48, 256), 2 * rng.randint(1, 4), "fp32",
                     rng.choice(["hllc", "hll"]), moving=moving, runs=rng.randint(3, 24))
    if kind == "remesh":
        return _case(None, kind, rng.choice(["tube", "shear"]), _log_int(rng, 32, 1000), 1, "fp32", solver, limiter)
    if kind == "plugins":
        return _case(None, kind, problem, _log_int(rng, 16, 512), 1, solver=solver, limiter=limiter,
                     reconstruction=rng.choice(["linear", "linear", "constant"]), moving=moving)
    precision = "fp32" if kind == "graph" else rng.choice(["fp32", "fp64"])
    side = _log_int(rng, 16, 1000 if precision == "fp32" else 700)
    steps = 2 * rng.randint(1, 5) if precision == "fp32" else rng.randint(1, 2)
    return _case(None, kind, problem, side, steps, precision, solver, limiter,
                 rng.choice(["linear", "linear", "linear", "constant"]), rng.random() < 0.85, moving)


# ---- inputs ---------------------------------------------------------------------------
def _problem(case, seed):
    """(host mesh, primitives of all cells): the problem, on its own jittered lattice, plus a
    smooth perturbation made from the seed."""
    side = case["side"]
    name = case["problem"]
    if name == "tube":
        mesh, prim, _ = pkg.problems.shock_tube(side)
    elif name == "explosion":
        mesh, prim, _ = pkg.problems.point_explosion(side)
        # the deposit spread to a finite radius over a warm background, as it looks once the
        # shock has run a while (the cold start's vacuum would not outlast a long timing)
        d = np.abs(mesh.x - 0.5)
        d = np.minimum(d, 1.0 - d)
        prim[3] = 0.1 + 2.0 * np.exp(-(d[0] ** 2 + d[1] ** 2) / (2.0 * 0.08 ** 2))
    elif name == "shear":
        mesh, prim, _ = pkg.problems.shear_layer(side)
    else:
        mesh, prim, _ = pkg.problems.gaussian_bump(side, background=False)
    return mesh, _perturbed(mesh, prim, np.random.default_rng(seed))


def _perturbed(mesh, prim, rng):
    x = mesh.x
    wave = np.zeros((4, x.shape[1]))
    for f in range(4):
        for _ in range(3):
            kx, ky = 2.0 * np.pi * rng.integers(1, 5, 2)
            wave[f] += rng.uniform(0.3, 1.0) * np.sin(kx * x[0] + rng.uniform(0, 6.28)) * \
                np.sin(ky * x[1] + rng.uniform(0, 6.28))
    prim = np.array(prim)
    prim[0] *= 1.0 + 0.02 * wave[0]
    prim[1] += 0.02 * wave[1]
    prim[2] += 0.02 * wave[2]
    prim[3] *= 1.0 + 0.02 * wave[3]
    return pkg.meshgen.fill_ghosts(mesh, prim)


def _stepper(case, mesh, prim):
    return pkg.FluxStepper(mesh, prim, gamma=GAMMA[case["problem"]], solver=case["solver"], limiter=case["limiter"],
                           reconstruction=case["reconstruction"], boost=case["boost"], moving=case["moving"],
                           precision=case["precision"])


def _ensemble_runs(case, seed):
    n = case["side"] ** 2
    rng = np.random.default_rng(seed)
    runs, _ = pkg.problems.riemann_ensemble(case["runs"], n_min=max(256, n // 64), n_max=n)
    return [(m, _perturbed(m, p, rng)) for m, p in runs]


def _bump_target(mesh):
    x = mesh.x[:, :mesh.n_real]
    return 1.0 + 0.1 * np.exp(-((x[0] - 0.4) ** 2 + (x[1] - 0.55) ** 2) / (2.0 * 0.05 ** 2))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        return dict(case=case, st=ensemble.EnsembleStepper(_ensemble_runs(case, seed), solver=case["solver"],
                                                           moving=case["moving"]))
    mesh, prim = _problem(case, seed)
    if kind == "plugins":
        it = (pkg.MovingMeshMUSCLHancock if case["moving"] else pkg.StaticMeshMUSCLHancock)()
        it.set_particles(pkg.HydroParticleCreator(num=mesh.n_cells, dim=2))
        it.set_domain_manager(pkg.DomainManager(list(mesh.xmin), list(mesh.xmax)))
        it.set_boundary_condition(pkg.Reflective() if mesh.boundary == "reflective" else pkg.Periodic())
        it.set_mesh(pkg.Mesh())
        it.set_reconstruction(pkg.PieceWiseLinear(limiter=case["limiter"]) if case["reconstruction"] == "linear"
                              else pkg.PieceWiseConstant())
        it.set_riemann({"hll": pkg.HLL, "hllc": pkg.HLLC, "exact": pkg.Exact}[case["solver"]](cfl=0.5))
        it.set_equation_state(pkg.IdealGas(GAMMA[case["problem"]]))
        it.initialize()
        it.before_loop(mesh, prim)
        return dict(case=case, it=it)
    st = _stepper(case, mesh, prim)
    state = dict(case=case, st=st)
    if kind == "graph":
        st.capture(case["steps"])
    elif kind == "remesh":
        state["pinned"] = st.dmesh.pinned_host_compact(mesh, resident=True)
        state["w_host"] = torch.empty((mesh.n_cells, 2), dtype=torch.float32, pin_memory=True)
    elif kind == "adjoint":
        recs = []
        for _ in range(case["steps"]):
            dt = st.read_clock().dt
            st.step(1)
            recs.append(adjoint.StepRecord(st.dmesh, st.face_w.clone(), dt))
        state["run"] = adjoint.FluxRunRecord(recs, gamma=GAMMA[case["problem"]], solver=case["solver"],
                                             limiter=case["limiter"], checkpoint=case["checkpoint"])
        state["prim0"] = torch.as_tensor(np.ascontiguousarray(prim[:, :mesh.n_real])).cuda()
        state["target"] = torch.as_tensor(_bump_target(mesh)).cuda()
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "plugins":
        it = state["it"]
        dt = it.compute_time_step()
        it.evolve_timestep()
        return {"cons": it.particles.block("conservative"), "prim": it.particles.block("primitive"), "dt": dt}
    if kind == "adjoint":
        p = state["prim0"].detach().requires_grad_(True)
        rho = adjoint.FluxRun.apply(p, state["run"])
        ((rho - state["target"]) ** 2).sum().backward()
        return {"rho": rho.detach(), "grad": p.grad}
    st = state["st"]
    if kind == "ensemble":
        st.step(case["steps"])
        return {"cons": st.cons, "prim": st.prim4, "dt": st.clocks.view(F64)[:, 0]}
    if kind == "graph":
        st.replay()
    elif kind == "remesh":
        st.load_mesh(state["pinned"])
        st.step_and_fetch(state["w_host"])
    else:
        st.step(case["steps"])
    out = {"cons": st.cons, "prim": st.prim4 if case["precision"] == "fp32" else st.prim,
           "dt": st.clock.buf.view(F64)[:1]}
    if kind == "remesh":
        out["w"] = state["w_host"]
    return out


def work(case):
    """A step reads each face's record (two cell ids, area, centroid offset, normal) and the
    cells' state, lists and geometry once and writes the state once: about 140 bytes a face
    in the fast precision, 152 in 64 bits, three faces to a cell; about 450 operations a
    face (states, wave speeds, flux) and 900 a cell (gradients, limiter, update).  A backward
    pass is counted as two steps; a hand-over brings 10 bytes a face from the host."""
    n = case["side"] ** 2
    if case["kind"] == "ensemble":           # sizes log-uniform between lo and n
        lo = max(256, n // 64)
        n = case["runs"] * ((n - lo) / math.log(n / lo) if n > lo else n)
    faces = 3 * n
    per = 140 if case["precision"] == "fp32" else 152
    passes = case["steps"] * (3 if case["kind"] == "adjoint" else 1)
    extra = 10 * faces + 8 * n if case["kind"] == "remesh" else 0
    return {"bytes": passes * per * faces + extra, "flops": passes * (450 * faces + 900 * n)}


# ---- the scheme in plain torch, 64 bits ---------------------------------------------------
class _Mesh:
    def __init__(self, m):
        def up(a, dt=F64):
            return torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device="cuda")
        self.n, self.nr = m.n_cells, m.n_real
        self.i, self.j, self.map = up(m.pair_i, torch.long), up(m.pair_j, torch.long), up(m.map, torch.long)
        self.x, self.dcom, self.vol = up(m.x), up(m.dcom), up(m.vol)
        self.area, self.com, self.normal = up(m.area), up(m.com), up(m.normal)
        ghost = np.arange(m.n_cells) >= m.n_real
        sign = np.ones((2, m.n_cells))
        if m.boundary == "reflective":           # a mirror ghost's normal velocity changes sign
            for k in range(2):
                sign[k, ghost & ((m.x[k] < m.xmin[k]) | (m.x[k] > m.xmax[k]))] = -1.0
        self.sign = up(sign)
        # both sides of each face; a real cell's gradient sums over its faces
        jr = self.j < self.nr
        f = torch.arange(self.i.numel(), device="cuda")
        self.c = torch.cat([self.i, self.j[jr]])
        self.o = torch.cat([self.j, self.i[jr]])
        self.f = torch.cat([f, f[jr]])
        self.jr = jr

    def all_cells(self, u):
        """Real rows -> all rows of a [mass-like, x, y, energy-like] field."""
        a = u[:, self.map]
        return torch.stack([a[0], a[1] * self.sign[0], a[2] * self.sign[1], a[3]])


def _nz(d):
    return torch.where(d == 0, torch.ones_like(d), d)


def _cons(q, vol, gamma):
    m = q[0] * vol
    return torch.stack([m, q[1] * m, q[2] * m, (0.5 * q[0] * (q[1] ** 2 + q[2] ** 2) + q[3] / (gamma - 1)) * vol])


def _prim(u, vol, gamma):
    vx, vy = u[1] / u[0], u[2] / u[0]
    rho = u[0] / vol
    return torch.stack([rho, vx, vy, (u[3] / vol - 0.5 * rho * (vx * vx + vy * vy)) * (gamma - 1)])


def _gradients(M, q, limiter):
    c, o, f, nr = M.c, M.o, M.f, M.nr
    r = M.x[:, c] - M.x[:, o]
    cf = M.com[:, f] - 0.5 * (M.x[:, c] + M.x[:, o])
    fac = M.area[f] / (torch.sqrt((r * r).sum(0)) * M.vol[c])
    qc, qo = q[:, c], q[:, o]
    g = torch.stack([torch.zeros((4, nr), dtype=F64, device=q.device).index_add(
        1, c, fac * ((qo - qc) * cf[k] - 0.5 * (qo + qc) * r[k])) for k in range(2)], 1)
    sep = M.com[:, f] - M.x[:, c] - M.dcom[:, c]
    dphi = g[:, 0, c] * sep[0] + g[:, 1, c] * sep[1]
    rows = c.expand(4, -1)
    one = torch.ones((4, nr), dtype=F64, device=q.device)
    if limiter == "arepo":
        hi = q[:, :nr].scatter_reduce(1, rows, qo, "amax")[:, c]
        lo = q[:, :nr].scatter_reduce(1, rows, qo, "amin")[:, c]
        psi = torch.where(dphi == 0, torch.ones_like(dphi), (torch.where(dphi > 0, hi, lo) - qc) / _nz(dphi))
        alpha = one.scatter_reduce(1, rows, psi.clamp(min=0), "amin")
    else:                                        # all fields limit the density's slope alone
        psi = torch.where(dphi == 0, torch.ones_like(dphi), ((qo - qc) / _nz(dphi)).clamp(min=0))
        alpha = torch.cat([one[:1].scatter_reduce(1, rows[:1], psi.amin(0, keepdim=True), "amin"), one[1:]])
    g = (alpha[:, None] * g)[:, :, M.map]        # [field][axis][cell]; ghosts take their image's
    flip = torch.ones((4, 2, M.n), dtype=F64, device=q.device)
    flip[1, 0], flip[2, 1] = M.sign[0], M.sign[1]
    return g * flip


def _pair_limit(sl, sr, qi, qj, ti, tj, L, R):
    """GIZMO's pair limiter: ti, tj the centroid distances over the cells' distance."""
    d = (sl - sr).abs()
    lo, hi = torch.minimum(sl, sr), torch.maximum(sl, sr)
    top = torch.where((hi + 0.5 * d) * hi >= 0, hi + 0.5 * d, hi / (1 + 0.5 * d / _nz(hi.abs())))
    bot = torch.where((lo - 0.5 * d) * lo >= 0, lo - 0.5 * d, lo / (1 + 0.5 * d / _nz(lo.abs())))
    ml, mr = sl + ti * (sr - sl), sr + tj * (sl - sr)
    up, down = qi < qj, qi > qj
    Lx = torch.where(up, torch.maximum(bot, torch.minimum(ml + 0.25 * d, L)),
                     torch.where(down, torch.minimum(top, torch.maximum(ml - 0.25 * d, L)), sl))
    Rx = torch.where(up, torch.minimum(top, torch.maximum(mr - 0.25 * d, R)),
                     torch.where(down, torch.maximum(bot, torch.minimum(mr + 0.25 * d, R)), sr))
    return Lx, Rx


def _states(M, q, g, w, dt, gamma, boost, linear):
    shift = torch.stack([torch.zeros_like(w[0]), w[0], w[1], torch.zeros_like(w[0])]) if boost else 0.0
    sides = []
    for c in (M.i, M.j):
        s = q[:, c] - shift
        sep = M.com - M.x[:, c] - M.dcom[:, c]
        sides.append((c, s, sep))
    (i, sl, si), (j, sr, sj) = sides
    if not linear:
        return sl, sr
    gi, gj = g[:, :, i], g[:, :, j]
    dist = torch.sqrt(((M.x[:, j] - M.x[:, i]) ** 2).sum(0))
    L, R = _pair_limit(sl, sr, q[:, i], q[:, j], torch.sqrt((si * si).sum(0)) / dist, torch.sqrt((sj * sj).sum(0)) / dist,
                       sl + (gi * si).sum(1), sr + (gj * sj).sum(1))
    out = []
    for X, c, s, gr in ((L, i, sl, gi), (R, j, sr, gj)):
        X = torch.where(((X[0] < 0) | (X[3] < 0))[None], s, X)
        p = q[:, c]
        v = s[1:3]                               # the cell's velocity in the states' frame
        adv = v[0] * gr[:, 0] + v[1] * gr[:, 1]
        div = gr[1, 0] + gr[2, 1]
        rate = torch.stack([adv[0] + p[0] * div, adv[1] + gr[3, 0] / p[0], adv[2] + gr[3, 1] / p[0],
                            adv[3] + gamma * p[3] * div])
        Y = X - 0.5 * dt * rate
        out.append(torch.where(((Y[0] < 0) | (Y[3] < 0))[None], X, Y))
    return out


def _waves(dl, ul, pl, dr, ur, pr, gamma):
    cl, cr = (gamma * pl / dl).sqrt().clamp(min=1e-10), (gamma * pr / dr).sqrt().clamp(min=1e-10)
    pv = (0.5 * (pl + pr) + 0.125 * (ul - ur) * (dl + dr) * (cl + cr)).clamp(min=0)
    lo, hi = torch.minimum(pl, pr), torch.maximum(pl, pr)
    z = (gamma - 1) / (2 * gamma)
    a = (pl / pr) ** z
    us = (a * ul / cl + ur / cr + 2 * (a - 1) / (gamma - 1)) / (a / cl + 1 / cr)
    tr = 0.5 * pl * (1 + (gamma - 1) * (ul - us) / (2 * cl)).clamp(min=1e-300) ** (1 / z) + \
        0.5 * pr * (1 + (gamma - 1) * (us - ur) / (2 * cr)).clamp(min=1e-300) ** (1 / z)
    b = (gamma - 1) / (gamma + 1)
    kl, kr = (2 / ((gamma + 1) * dl * (pv + b * pl))).sqrt(), (2 / ((gamma + 1) * dr * (pv + b * pr))).sqrt()
    ts = (kl * pl + kr * pr - (ur - ul)) / (kl + kr)
    ps = torch.where((hi < 2 * lo) & (lo < pv) & (pv < hi), pv, torch.where(pv <= lo, tr, ts))
    k = (gamma + 1) / (2 * gamma)
    sl = ul - cl * torch.where(ps <= pl, torch.ones_like(ps), (1 + k * (ps / pl - 1)).clamp(min=1e-300).sqrt())
    sr = ur + cr * torch.where(ps <= pr, torch.ones_like(ps), (1 + k * (ps / pr - 1)).clamp(min=1e-300).sqrt())
    sc = (pr - pl + dl * ul * (sl - ul) - dr * ur * (sr - ur)) / _nz(dl * (sl - ul) - dr * (sr - ur))
    return sl, sc, sr


def _exact_star(dl, ul, pl, cl, dr, ur, pr, cr, gamma):
    """p* and u* of the exact Riemann problem, Newton to convergence (p* held fixed for autograd,
    then one differentiable Newton step, which carries the implicit derivative)."""
    def side(p, d, pk, c):
        A, B = 2 / ((gamma + 1) * d), pk * (gamma - 1) / (gamma + 1)
        q = (p / pk).clamp(min=1e-300)
        rare = p <= pk
        s = (A / (p + B)).sqrt()
        f = torch.where(rare, 2 * c / (gamma - 1) * (q ** ((gamma - 1) / (2 * gamma)) - 1), (p - pk) * s)
        df = torch.where(rare, q ** (-(gamma + 1) / (2 * gamma)) / (d * c), s * (1 - 0.5 * (p - pk) / (B + p)))
        return f, df
    with torch.no_grad():
        p = 0.5 * (pl + pr) - 0.125 * (ur - ul) * (dl + dr) * (cl + cr)
        p = torch.maximum(p, 1e-3 * torch.minimum(pl, pr))
        for _ in range(60):
            (fl, dfl), (fr, dfr) = side(p, dl, pl, cl), side(p, dr, pr, cr)
            step = (fl + fr + ur - ul) / (dfl + dfr)
            p = torch.maximum(p - step, 0.1 * p)
    (fl, dfl), (fr, dfr) = side(p, dl, pl, cl), side(p, dr, pr, cr)
    p = p - (fl + fr + ur - ul) / (dfl + dfr).detach()
    fl, fr = side(p, dl, pl, cl)[0], side(p, dr, pr, cr)[0]
    return p, 0.5 * (ul + ur + fr - fl)


def _exact_flux(L, R, n, gamma):
    ul, ur = (L[1:3] * n).sum(0), (R[1:3] * n).sum(0)
    cl, cr = (gamma * L[3] / L[0]).sqrt(), (gamma * R[3] / R[0]).sqrt()
    ps, us = _exact_star(L[0], ul, L[3], cl, R[0], ur, R[3], cr, gamma)
    left = us >= 0
    sg = torch.where(left, 1.0, -1.0).to(F64)    # the right side is the left one mirrored
    S = torch.where(left[None], L, R)
    d, p, c = S[0], S[3], torch.where(left, cl, cr)
    u, us = sg * torch.where(left, ul, ur), sg * us
    g1, gp = gamma - 1, gamma + 1
    q = ps / p
    shock = ps > p
    cs = c * q ** (g1 / (2 * gamma))
    fan_c = 2 / gp * (c + 0.5 * g1 * u)
    fr = (fan_c / c).clamp(min=1e-300)
    head = torch.where(shock, u - c * (gp / (2 * gamma) * q + g1 / (2 * gamma)).sqrt(), u - c)
    fan = ~shock & (us - cs > 0)
    ds = torch.where(shock, d * (q + g1 / gp) / (g1 / gp * q + 1), d * q ** (1 / gamma))
    data = head >= 0
    d2 = torch.where(data, d, torch.where(fan, d * fr ** (2 / g1), ds))
    p2 = torch.where(data, p, torch.where(fan, p * fr ** (2 * gamma / g1), ps))
    u2 = torch.where(data, u, torch.where(fan, fan_c, us))
    v = S[1:3] + sg * (u2 - u) * n
    vn = sg * u2
    e = 0.5 * d2 * (v * v).sum(0) + gamma * p2 / g1
    return torch.stack([d2 * vn, d2 * v[0] * vn + p2 * n[0], d2 * v[1] * vn + p2 * n[1], e * vn])


def _flux(M, L, R, w, gamma, solver, boost):
    n = M.normal
    if solver == "exact":
        f = _exact_flux(L, R, n, gamma)
    else:
        wn = torch.zeros_like(L[0]) if boost else (w * n).sum(0)
        ul, ur = (L[1:3] * n).sum(0), (R[1:3] * n).sum(0)
        sl, sc, sr = _waves(L[0], ul, L[3], R[0], ur, R[3], gamma)

        def side(S, u):
            e = 0.5 * S[0] * (S[1] ** 2 + S[2] ** 2) + S[3] / (gamma - 1)
            U = torch.stack([S[0], S[0] * S[1], S[0] * S[2], e])
            zero = torch.zeros_like(u)
            return U, U * u + torch.stack([zero, S[3] * n[0], S[3] * n[1], S[3] * u])
        (Ul, Fl), (Ur, Fr) = side(L, ul), side(R, ur)
        if solver == "hll":
            mid = (Fl * (sr - wn) - Fr * (sl - wn) - sl * Ul * (sr - wn) + sr * Ur * (sl - wn)) / _nz(sr - sl)
        else:
            def star(S, U, F, u, s):
                k = S[0] * (s - u) / _nz(s - sc)
                e = U[3] / S[0] + (sc - u) * (sc + S[3] / _nz(S[0] * (s - u)))
                V = torch.stack([k, k * (S[1] + (sc - u) * n[0]), k * (S[2] + (sc - u) * n[1]), k * e])
                return F + s * (V - U) - wn * V
            mid = torch.where((wn <= sc)[None], star(L, Ul, Fl, ul, sl), star(R, Ur, Fr, ur, sr))
        f = torch.where((wn <= sl)[None], Fl - wn * Ul, torch.where((wn <= sr)[None], mid, Fr - wn * Ur))
    if boost or solver == "exact":
        f = torch.stack([f[0], f[1] + w[0] * f[0], f[2] + w[1] * f[0],
                         f[3] + w[0] * f[1] + w[1] * f[2] + 0.5 * (w[0] ** 2 + w[1] ** 2) * f[0]])
    return f


def _face_velocity(M, q, gamma, eta=0.25):
    c = (gamma * q[3] / q[0]).sqrt()
    d = torch.sqrt((M.dcom ** 2).sum(0))
    eR = eta * torch.sqrt(M.vol / math.pi)
    k = torch.where(d < 0.9 * eR, torch.zeros_like(d),
                    torch.where(d < 1.1 * eR, c * (d - 0.9 * eR) / (0.2 * eR), c) / _nz(d))
    v = q[1:3] + k * M.dcom
    wi, wj = v[:, M.i], v[:, M.j]
    dx = M.x[:, M.j] - M.x[:, M.i]
    off = M.com - 0.5 * (M.x[:, M.i] + M.x[:, M.j])
    return v, 0.5 * (wi + wj) + ((wi - wj) * off).sum(0) / (dx * dx).sum(0) * dx


def _time_step(M, q, gamma, boost):
    q = q[:, :M.nr]
    c = (gamma * q[3] / q[0]).sqrt()
    return torch.sqrt(M.vol[:M.nr] / math.pi) / (c if boost else c + torch.sqrt(q[1] ** 2 + q[2] ** 2))


def _advance(M, case, u, q, w, dt, gamma):
    """Real cells' totals after one step; dt a number or one value a face."""
    boost, linear = case["boost"] or case["solver"] == "exact", case["reconstruction"] == "linear"
    g = _gradients(M, q, case["limiter"]) if linear else None
    L, R = _states(M, q, g, w, dt, gamma, boost, linear)
    inc = dt * M.area * _flux(M, L, R, w, gamma, case["solver"], boost)
    return u[:, :M.nr].index_add(1, M.i, -inc).index_add(1, M.j[M.jr], inc[:, M.jr])


def exact(case, seed):
    kind = case["kind"]
    gamma = GAMMA.get(case["problem"], 1.4)
    boost = case["boost"] or case["solver"] == "exact"
    if kind == "ensemble":
        runs = _ensemble_runs(case, seed)
        host, run_of, _, _ = ensemble.concatenate([m for m, _ in runs])
        nr = host.n_real
        real = np.concatenate([p[:, :m.n_real] for m, p in runs], axis=1)
        M = _Mesh(host)
        q = M.all_cells(torch.as_tensor(real).cuda())
        rows = torch.as_tensor(run_of).long().cuda()
    else:
        mesh, prim = _problem(case, seed)
        M = _Mesh(mesh)
        q = torch.as_tensor(prim).cuda()

    def step_of(q):
        cand = 0.5 * _time_step(M, q, gamma, boost)
        if kind != "ensemble":
            return cand.min(), cand.min()
        dt = torch.full((case["runs"],), math.inf, dtype=F64, device="cuda").scatter_reduce(0, rows[:nr], cand, "amin")
        return dt, dt[rows[M.i]]

    if kind == "adjoint":
        p0 = q[:, :M.nr].clone().requires_grad_(True)
        u = _cons(p0, M.vol[:M.nr], gamma)
        for _ in range(case["steps"]):
            qa = _prim(M.all_cells(u), M.vol, gamma)
            with torch.no_grad():                # dt and the face velocities are held fixed
                dt = step_of(qa)[1]
                w = _face_velocity(M, qa, gamma)[1] if case["moving"] else torch.zeros_like(M.com)
            u = checkpoint(lambda uu, ww, d: _advance(M, case, uu, _prim(M.all_cells(uu), M.vol, gamma), ww, d, gamma),
                           u, w, dt, use_reentrant=False)
        rho = u[0] / M.vol[:M.nr]
        ((rho - torch.as_tensor(_bump_target(mesh)).cuda()) ** 2).sum().backward()
        return {"rho": rho.detach(), "grad": p0.grad}
    with torch.no_grad():
        ua = _cons(q, M.vol, gamma)
        for _ in range(case["steps"]):
            dts, dt = step_of(q)
            v, w = _face_velocity(M, q, gamma)
            if not case["moving"]:
                w = torch.zeros_like(w)
            ua = M.all_cells(_advance(M, case, ua, q, w, dt, gamma))
            q = _prim(ua, M.vol, gamma)
        if kind == "plugins":                    # a plugin step reports the dt it took
            return {"cons": ua, "prim": q, "dt": float(dts)}
        out = {"cons": ua, "prim": q.t().contiguous() if case["precision"] == "fp32" else q}
        out["dt"] = step_of(q)[0].reshape(-1)
        if kind == "remesh":
            out["w"] = v.t().contiguous()
        return out
