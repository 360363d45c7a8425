"""Hand-written adjoint of the flux path behind a ``torch.autograd.Function``.

The differentiable map is one run of steps ``U_{n+1} = step(U_n; mesh_n, w_n, dt_n)``
on the real cells' conserved totals, with each step's mesh (geometry and neighbour
lists), face velocities and time step recorded from a forward run and held fixed --
the tessellation, the mesh motion and the CFL choice are not differentiated.  The
backward pass runs the reverse-mode kernels of ``phd_adj.cu`` step by step, from the
last step to the first, recomputing each segment's states from checkpoints taken
every ``checkpoint`` steps (checkpoint-and-recompute: memory holds the checkpoints and
one segment).

``FluxRun.apply(prim0, run)`` maps the real cells' initial primitives ``[4][n_real]``
(rho, v_x, v_y, p) to the final densities ``[n_real]``; gradients flow back to
``prim0``.
"""
import ctypes
import weakref

import numpy as np
import torch

from . import _lib as L
from .device import DeviceClock, DeviceMesh, make_params

F64 = torch.float64


def adjoint_index(host):
    """Partner entries and per-image ghost lists of a host mesh (numpy int32)."""
    ptr, idx = host.nbr_ptr, host.nbr_idx
    E = int(ptr[-1])
    cells = np.repeat(np.arange(host.n_cells), np.diff(ptr))
    faces = idx[:E]
    o = np.lexsort((cells, faces))              # entries grouped by face, two per face
    partner = np.full(E, -1, dtype=np.int32)
    fa = faces[o]
    same = fa[0::2] == fa[1::2]
    if not np.all(same):
        raise RuntimeError("every face must appear in exactly two cells' lists")
    a, b = o[0::2], o[1::2]
    partner[a] = b
    partner[b] = a
    g = np.arange(host.n_real, host.n_cells)
    img = host.map[g]
    og = np.argsort(img, kind="stable")
    ghost_idx = g[og].astype(np.int32)
    cnt = np.bincount(img, minlength=host.n_real)
    ghost_ptr = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int32)
    return partner, ghost_ptr, ghost_idx


class StepRecord:
    """What one step holds fixed: its device mesh, face velocities and dt."""

    def __init__(self, dmesh, face_w, dt):
        self.dmesh = dmesh
        self.face_w = face_w
        self.dt = float(dt)

    def index(self):
        """Partner/ghost index of the step's mesh, built once per device mesh."""
        dm = self.dmesh
        cached = getattr(dm, "_adjoint_index", None)
        if cached is None:
            p, gp, gi = adjoint_index(dm.host)
            tens = [torch.as_tensor(a).to(dm.device) for a in (p, gp, gi)]
            cached = (tens, L.PhdAdjIndex(*(t.data_ptr() for t in tens)))
            dm._adjoint_index = cached
        return cached[1]


class _MeshBuffers:
    """Per-mesh device buffers reused by every step on that mesh."""

    def __init__(self, dm, device):
        n, F = dm.n_cells, max(dm.n_faces, 1)
        self.cons = torch.zeros((4, n), dtype=F64, device=device)
        self.nxt = torch.zeros_like(self.cons)
        self.prim = torch.zeros_like(self.cons)
        self.grad = torch.zeros((8, n), dtype=F64, device=device)
        self.w = torch.zeros((2, n), dtype=F64, device=device)
        self.flux = torch.zeros((4, F), dtype=F64, device=device)
        self.lam_next = torch.zeros_like(self.cons)      # ghost rows stay zero
        self.lam = torch.zeros_like(self.cons)
        self.work = None

    def adjoint_work(self, lib, dm, device):
        if self.work is None:
            self.work = torch.empty(int(lib.phd_adjoint_work_doubles(dm.n_cells, dm.n_faces)), dtype=F64,
                                    device=device)
        return self.work


class _Tail:
    """The last segment's states from a forward pass that kept them, for one backward pass."""

    def __init__(self, states):
        self.states = states

    def take(self):
        states, self.states = self.states, None
        return states


class FluxRunRecord:
    """A recorded run: the per-step records and the options of the step.

    Consecutive steps on the same device mesh are chained on the device: the update
    kernel already writes the next step's totals and primitives for every cell, ghosts
    included, so only a change of mesh goes back through the real cells (ghost refresh
    and primitive recovery on the new mesh).  Each step owns a row of a device clock
    table (its dt), so no step waits on the host.
    """

    def __init__(self, steps, gamma=1.4, solver="hllc", limiter="arepo", gizmo=True, boost=True,
                 reconstruction="linear", checkpoint=20, final_vol=None):
        if solver not in ("hll", "hllc", "exact"):
            raise ValueError("solver must be 'hll', 'hllc' or 'exact'")
        self.steps = steps
        self.params = make_params(gamma=gamma, solver=solver, limiter=limiter, gizmo=gizmo, boost=boost,
                                  reconstruction=reconstruction)
        self.checkpoint = max(1, int(checkpoint))
        self.final_vol = final_vol if final_vol is not None else steps[-1].dmesh.vol[:steps[-1].dmesh.n_real]
        d0 = steps[0].dmesh
        self.device = d0.device
        self.n_real = d0.n_real
        self.clock = DeviceClock(self.device)
        rows = []
        for rec in steps:
            c = L.PhdClock()
            c.dt = rec.dt
            c.dtmin_bits = np.float64(np.inf).view(np.uint64).item()
            rows.append(np.frombuffer(bytes(c), dtype=np.uint8))
        self._clocks0 = torch.as_tensor(np.stack(rows)).to(self.device)
        self.clocks = self._clocks0.clone()
        self._bufs = {}
        self._kept = None                    # the _Tail of a forward pass asked to keep one
        self._kept_ref = None                # and that of the newest pass, whoever holds it

    @property
    def _tail(self):
        """The newest forward pass's last segment while it is held and not yet used."""
        kept = self._kept_ref() if self._kept_ref is not None else None
        return None if kept is None else kept.states

    def _buffers(self, dm):
        b = self._bufs.get(id(dm))
        if b is None:
            b = self._bufs[id(dm)] = _MeshBuffers(dm, self.device)
        return b

    def _clock_ptr(self, k):
        return ctypes.c_void_p(self.clocks[k].data_ptr())

    def _load_real(self, dm, U_real, cons, prim):
        """All-cell totals and primitives on mesh dm from the real cells' totals."""
        s = L.stream_handle()
        lib = L.lib()
        cons[:, :dm.n_real].copy_(U_real)
        L.check(lib.phd_ghost_cons_f64(dm.ref, L.ptr(cons), s), "ghost")
        L.check(lib.phd_prim_from_cons_f64(2, dm.n_cells, self.params.gamma, L.ptr(dm.vol), L.ptr(cons),
                                           L.ptr(prim), s), "prim")

    def _step(self, k, prim, cons, nxt, grad, tape=None):
        """Step k: prim is overwritten with the next primitives, nxt receives the next
        totals (all cells), grad the limited gradients of the incoming primitives and,
        with a tape (f64, i32), the limiter's record for the adjoint."""
        rec = self.steps[k]
        b = self._buffers(rec.dmesh)
        lib = L.lib()
        if tape is None:
            L.check(lib.phd_step_f64(rec.dmesh.ref, ctypes.byref(self.params), 0, L.ptr(prim), L.ptr(cons),
                                     L.ptr(nxt), L.ptr(grad), L.ptr(b.w), L.ptr(rec.face_w), L.ptr(b.flux),
                                     self._clock_ptr(k), L.stream_handle()), "step")
        else:
            L.check(lib.phd_step_f64_taped(rec.dmesh.ref, ctypes.byref(self.params), 0, L.ptr(prim), L.ptr(cons),
                                           L.ptr(nxt), L.ptr(grad), L.ptr(b.w), L.ptr(rec.face_w), L.ptr(b.flux),
                                           L.ptr(tape[0]), L.ptr(tape[1]), self._clock_ptr(k),
                                           L.stream_handle()), "step")

    # --- one step in isolation, on real-cell totals (tests use these) ---------------
    def _forward_step(self, rec, U_real):
        dm = rec.dmesh
        cons = torch.zeros((4, dm.n_cells), dtype=F64, device=self.device)
        prim, nxt = torch.empty_like(cons), torch.empty_like(cons)
        grad = torch.zeros((8, dm.n_cells), dtype=F64, device=self.device)
        self._load_real(dm, U_real, cons, prim)
        self.clock.set(dt=rec.dt)
        b = self._buffers(dm)
        L.check(L.lib().phd_step_f64(dm.ref, ctypes.byref(self.params), 0, L.ptr(prim), L.ptr(cons), L.ptr(nxt),
                                     L.ptr(grad), L.ptr(b.w), L.ptr(rec.face_w), L.ptr(b.flux), self.clock.ptr,
                                     L.stream_handle()), "step")
        return nxt[:, :dm.n_real].clone()

    def _adjoint_step(self, rec, U_real, lam_next_real):
        dm = rec.dmesh
        cons = torch.zeros((4, dm.n_cells), dtype=F64, device=self.device)
        prim = torch.empty_like(cons)
        grad = torch.zeros((8, dm.n_cells), dtype=F64, device=self.device)
        self._load_real(dm, U_real, cons, prim)
        if self.params.reconstruction == L.LINEAR:
            L.check(L.lib().phd_gradients_f64(dm.ref, L.ptr(prim), self.params.limiter, L.ptr(grad), self.clock.ptr,
                                              L.stream_handle()), "gradients")
        return self._adjoint(rec, (cons, prim, grad, None), lam_next_real)

    def _adjoint(self, rec, state, lam_next_real):
        """lam_n (real cells) from lam_{n+1} at the step's recorded all-cell state
        (cons, prim, grad, tape); with a limiter tape the reverse reads the forward's
        selections instead of recomputing them."""
        dm = rec.dmesh
        b = self._buffers(dm)
        b.lam_next[:, :dm.n_real].copy_(lam_next_real)
        self._reverse(rec, state, b)
        return b.lam[:, :dm.n_real].clone()

    def _reverse(self, rec, state, b):
        """b.lam from b.lam_next (all cells, ghost rows zero in both)."""
        cons, prim, grad, tape = state
        dm = rec.dmesh
        lib = L.lib()
        common = (dm.ref, ctypes.byref(rec.index()), ctypes.byref(self.params), rec.dt, L.ptr(cons), L.ptr(prim),
                  L.ptr(grad), L.ptr(rec.face_w), L.ptr(b.lam_next), L.ptr(b.lam),
                  L.ptr(b.adjoint_work(lib, dm, self.device)))
        if tape is None:
            L.check(lib.phd_adjoint_step_f64(*common, L.stream_handle()), "phd_adjoint_step_f64")
        else:
            L.check(lib.phd_adjoint_step_f64_taped(*common, L.ptr(tape[0]), L.ptr(tape[1]), L.stream_handle()),
                    "phd_adjoint_step_f64_taped")

    # --- whole run ------------------------------------------------------------------
    def _tail_start(self):
        """First step of the last segment where its states may be kept from the forward pass
        to the backward one, else the number of steps.  They take no more than the
        backward pass takes for them anyway, but they are held in between: up to a 64th of
        the device's memory, past which (16 million cell-steps) the segment is recomputed."""
        N = len(self.steps)
        a = (N - 1) // self.checkpoint * self.checkpoint
        rows = 8 * (4 + 4 + 8 + L.GRAD_TAPE_F64_ROWS) + 4 * L.GRAD_TAPE_I32_ROWS
        cells = sum(rec.dmesh.n_cells for rec in self.steps[a:])
        return a if rows * cells <= torch.cuda.get_device_properties(self.device).total_memory // 64 else N

    def forward(self, U0, keep=False):
        """Run all steps from U0 [4][n_real]; keep checkpoints; return U_T.  With ``keep`` the
        last segment is recorded as it runs, for the next ``backward``: its recomputation was
        a sixth of a pass over two segments (12.4 -> 10.8 ms, 40 steps at 128 x 128)."""
        self.clocks.copy_(self._clocks0)
        self.ckpt = {0: U0.clone()}
        self._kept = self._kept_ref = None
        N = len(self.steps)
        tail = self._tail_start() if keep else N
        prev = kept = None
        for k, rec in enumerate(self.steps):
            dm = rec.dmesh
            b = self._buffers(dm)
            if prev is None:
                self._load_real(dm, U0, b.cons, b.prim)
            elif prev is not b:
                self._load_real(dm, prev.cons[:, :dm.n_real], b.cons, b.prim)
            if k == tail:
                states, cons = self._segment(k, N, b.cons.clone(), b.prim.clone(), True)
                kept = _Tail(states)
                break
            self._step(k, b.prim, b.cons, b.nxt, b.grad)
            b.cons, b.nxt = b.nxt, b.cons
            prev = b
            cons = b.cons
            if (k + 1) % self.checkpoint == 0 and k + 1 < N:
                self.ckpt[k + 1] = b.cons[:, :dm.n_real].clone()
        UT = cons[:, :self.steps[-1].dmesh.n_real].clone()
        st = 0
        for row in self.clocks.cpu().numpy():
            st |= L.PhdClock.from_buffer_copy(row.tobytes()).status
        L.raise_status(st)
        if kept is not None:
            self._kept, self._kept_ref = kept, weakref.ref(kept)
        return UT

    # --- branch-frozen forward (finite differences on the branch the run takes) ----
    def forward_frozen(self, U0, record):
        """U_T from U0 through phd_step_f64_frozen.  With ``record`` the run from U0 is
        the ordinary forward, and every step's limiter selections and face decisions are
        written to this run's tapes; without it they are read back, so U0 -> U_T is the
        smooth map of the recorded run's branches, whose derivative the adjoint
        computes -- central differences through it check the adjoint even where the
        limited scheme itself has kinks within the difference step."""
        lib = L.lib()
        if record or getattr(self, "_frozen", None) is None:
            if not record:
                raise RuntimeError("forward_frozen: record a run before replaying it")
            self._frozen = []
            for rec in self.steps:
                dm = rec.dmesh
                self._frozen.append((torch.empty((L.GRAD_TAPE_F64_ROWS, dm.n_cells), dtype=F64, device=self.device),
                                     torch.empty((L.GRAD_TAPE_I32_ROWS, dm.n_cells), dtype=torch.int32,
                                                 device=self.device),
                                     torch.zeros(max(dm.n_faces, 1), dtype=torch.int64, device=self.device)))
        self.clock.set(dt=self.steps[0].dt)
        mode = L.FROZEN_RECORD if record else L.FROZEN_REPLAY
        prev = None
        for k, rec in enumerate(self.steps):
            dm = rec.dmesh
            b = self._buffers(dm)
            if prev is None:
                self._load_real(dm, U0, b.cons, b.prim)
            elif prev is not b:
                self._load_real(dm, prev.cons[:, :dm.n_real], b.cons, b.prim)
            tf, ti, fb = self._frozen[k]
            L.check(lib.phd_step_f64_frozen(dm.ref, ctypes.byref(self.params), mode, rec.dt, L.ptr(b.prim),
                                            L.ptr(b.cons), L.ptr(b.nxt), L.ptr(b.grad), L.ptr(rec.face_w),
                                            L.ptr(b.flux), L.ptr(tf), L.ptr(ti), L.ptr(fb), self.clock.ptr,
                                            L.stream_handle()), "phd_step_f64_frozen")
            b.cons, b.nxt = b.nxt, b.cons
            prev = b
        self.clock.check_status()
        return prev.cons[:, :self.steps[-1].dmesh.n_real].clone()

    def final_density_frozen(self, prim0, record=False):
        """Final densities [n_real] from the real cells' initial primitives through the
        branch-frozen forward (see forward_frozen)."""
        vol0 = self.steps[0].dmesh.vol[:self.n_real]
        U0 = cons_from_prim_t(prim0, vol0, self.params.gamma)
        return self.forward_frozen(U0.contiguous(), record)[0] / self.final_vol

    def _loaded(self, dm, U_real):
        """Totals and primitives (new tensors, all cells) on mesh dm from the real cells' totals."""
        c = torch.empty((4, dm.n_cells), dtype=F64, device=self.device)
        p = torch.empty_like(c)
        self._load_real(dm, U_real, c, p)
        return c, p

    def _replay_segment(self, a, b, ckpt=None):
        """Recompute the all-cell states entering steps a..b-1 from the checkpoint at a."""
        self.clocks[a:b].copy_(self._clocks0[a:b])      # each step's CFL finish overwrote its dt
        return self._segment(a, b, *self._loaded(self.steps[a].dmesh, (self.ckpt if ckpt is None else ckpt)[a]))[0]

    def _segment(self, a, b, cons, prim, finish=False):
        """The all-cell states (totals, primitives, gradients and the gradients' limiter tape)
        entering steps a..b-1 from the first ones, and with ``finish`` the totals after them."""
        states = []
        lib = L.lib()
        for k in range(a, b):
            dm = self.steps[k].dmesh
            n = dm.n_cells
            if k > a and self.steps[k - 1].dmesh is not dm:
                cons, prim = self._loaded(dm, cons[:, :dm.n_real])
            tape = None
            if self.params.reconstruction != L.LINEAR:
                grad = torch.zeros((8, n), dtype=F64, device=self.device)
            else:
                grad = torch.empty((8, n), dtype=F64, device=self.device)
                tape = (torch.empty((L.GRAD_TAPE_F64_ROWS, n), dtype=F64, device=self.device),
                        torch.empty((L.GRAD_TAPE_I32_ROWS, n), dtype=torch.int32, device=self.device))
            states.append((cons, prim, grad, tape))
            if finish or k + 1 < b:
                nxt = torch.empty_like(cons)
                p_next = prim.clone()                   # the step overwrites its primitives
                self._step(k, p_next, cons, nxt, grad, tape)
                cons, prim = nxt, p_next
            elif tape is not None:
                L.check(lib.phd_gradients_f64_taped(dm.ref, L.ptr(prim), self.params.limiter, L.ptr(grad),
                                                    L.ptr(tape[0]), L.ptr(tape[1]), self._clock_ptr(k),
                                                    L.stream_handle()), "gradients")
        return states, cons

    def backward(self, lam_T, ckpt=None, kept=None):
        """dLoss/dU_0 from dLoss/dU_T, segment by segment (recompute from checkpoints): of the
        newest forward pass, or of the one whose checkpoints and kept segment are given."""
        lam = lam_T
        if ckpt is None:
            ckpt, kept = self.ckpt, self._kept
        N = len(self.steps)
        prev = None                                     # the buffers whose lam is current
        starts = sorted(ckpt)
        for si in range(len(starts) - 1, -1, -1):
            a = starts[si]
            b = starts[si + 1] if si + 1 < len(starts) else N
            states = kept.take() if b == N and kept is not None else None
            if states is None:
                states = self._replay_segment(a, b, ckpt)
            for k in range(b - 1, a - 1, -1):
                rec = self.steps[k]
                bufs = self._buffers(rec.dmesh)
                if prev is bufs:                        # the same mesh: lam is the next step's lam_next as it stands
                    bufs.lam, bufs.lam_next = bufs.lam_next, bufs.lam
                else:
                    bufs.lam_next[:, :rec.dmesh.n_real].copy_(lam if prev is None else prev.lam[:, :rec.dmesh.n_real])
                self._reverse(rec, states[k - a], bufs)
                prev = bufs
            del states
        return prev.lam[:, :self.steps[0].dmesh.n_real].clone()


def cons_from_prim_t(prim, vol, gamma):
    m = prim[0] * vol
    return torch.stack([m, prim[1] * m, prim[2] * m,
                        (0.5 * prim[0] * (prim[1] ** 2 + prim[2] ** 2) + prim[3] / (gamma - 1.0)) * vol])


class FluxRun(torch.autograd.Function):
    """prim0 [4][n_real] -> final densities [n_real] through a recorded run.

    A pass's checkpoints and kept segment go with its graph, so that each backward pass is of
    its own forward pass, and what a graph held is given back with it."""

    @classmethod
    def apply(cls, prim0, run):
        # in forward the grad mode is off and needs_input_grad is the leaf's own, with or
        # without no_grad: asked here
        return super().apply(prim0, run, torch.is_grad_enabled())

    @staticmethod
    def forward(ctx, prim0, run, grad_mode):
        vol0 = run.steps[0].dmesh.vol[:run.n_real]
        with torch.no_grad():
            U0 = cons_from_prim_t(prim0, vol0, run.params.gamma)
            UT = run.forward(U0.contiguous(), keep=grad_mode and ctx.needs_input_grad[0])
        ctx.run, ctx.ckpt, ctx.kept = run, run.ckpt, run._kept
        run._kept = None                                # the graph's alone
        ctx.save_for_backward(prim0)
        return UT[0] / run.final_vol

    @staticmethod
    def backward(ctx, g_rho):
        run = ctx.run
        (prim0,) = ctx.saved_tensors
        lam_T = torch.zeros((4, run.n_real), dtype=F64, device=prim0.device)
        lam_T[0] = g_rho / run.final_vol
        lam0 = run.backward(lam_T, ctx.ckpt, ctx.kept)
        vol0 = run.steps[0].dmesh.vol[:run.n_real]
        # cons_from_prim is local and smooth: its vector-Jacobian product via autograd
        with torch.enable_grad():
            p = prim0.detach().requires_grad_(True)
            U = cons_from_prim_t(p, vol0, run.params.gamma)
            (gp,) = torch.autograd.grad(U, p, grad_outputs=lam0)
        return gp, None, None
