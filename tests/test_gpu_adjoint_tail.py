"""A differentiated run keeps its last segment's states from the forward pass: the gradient is
that of the recomputed segment bit for bit, a second backward pass recomputes it, and where
the states would hold too much memory none are kept."""
import numpy as np
import pytest
import torch

import phd_code_gb300 as pkg
from phd_code_gb300.adjoint import FluxRun, FluxRunRecord, StepRecord, cons_from_prim_t

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps, checkpoint", [(1, 20), (5, 20), (6, 3), (7, 3), (5, 1)])
@pytest.mark.parametrize("limiter, reconstruction", [("arepo", "linear"), ("tess", "linear"), ("arepo", "constant")])
def test_kept_segment(steps, checkpoint, limiter, reconstruction, monkeypatch):
    mesh, prim, _ = pkg.problems.gaussian_bump(16, background=False)
    st = pkg.FluxStepper(mesh, prim, gamma=1.4, limiter=limiter, reconstruction=reconstruction, moving=True)
    recs = []
    for _ in range(steps):
        dt = st.read_clock().dt
        st.step(1)
        recs.append(StepRecord(st.dmesh, st.face_w.clone(), dt))
    run = FluxRunRecord(recs, gamma=1.4, limiter=limiter, reconstruction=reconstruction, checkpoint=checkpoint)
    p0 = torch.tensor(prim[:, :mesh.n_real], device="cuda")
    lam = torch.tensor(np.random.default_rng(1).standard_normal(mesh.n_real), device="cuda")

    def gradient(retain=False):
        p = p0.clone().requires_grad_(True)
        rho = FluxRun.apply(p, run)
        assert (run._tail is None) == (run._tail_start() == steps)
        rho.backward(lam, retain_graph=retain)
        first, p.grad = p.grad, None
        if retain:
            rho.backward(lam)
            assert torch.equal(first, p.grad)
        return rho.detach(), first

    rho, g = gradient(retain=True)
    assert run._tail is None
    U0 = cons_from_prim_t(p0, mesh_vol := recs[0].dmesh.vol[:mesh.n_real], 1.4).contiguous()
    assert torch.equal(rho, run.forward(U0)[0] / mesh_vol) and run._tail is None
    monkeypatch.setattr(FluxRunRecord, "_tail_start", lambda self: steps)
    rho_r, g_r = gradient()
    assert torch.equal(rho, rho_r) and torch.equal(g, g_r) and bool(torch.isfinite(g).all())
