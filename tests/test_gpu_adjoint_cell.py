"""The reverse of the limited gradients by four threads a cell (taped forward step) against the
kernel with a thread a cell that recomputes the limiter's selections: ghosts with
reflective flips, lists longer than a quad's round, meshes that end within a block."""
import numpy as np
import pytest
import torch

import phd_code_gb300 as pkg
from _util import lattice_mesh, smooth_state
from phd_code_gb300.adjoint import FluxRunRecord, StepRecord, cons_from_prim_t

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limiter", ["arepo", "tess"])
@pytest.mark.parametrize("side, boundary", [(4, "reflective"), (5, "periodic"), (11, "reflective"), (17, "periodic")])
def test_quads_equal_one_thread_a_cell(side, boundary, limiter):
    mesh = lattice_mesh(side, boundary, seed=6)
    prim = smooth_state(mesh)
    st = pkg.FluxStepper(mesh, prim, gamma=1.4, limiter=limiter, moving=True)
    dt = st.read_clock().dt
    st.step(1)
    rec = StepRecord(st.dmesh, st.face_w.clone(), dt)
    run = FluxRunRecord([rec], gamma=1.4, limiter=limiter)
    U0 = cons_from_prim_t(torch.tensor(prim[:, :mesh.n_real], device="cuda"), rec.dmesh.vol[:mesh.n_real], 1.4)
    run.forward(U0.contiguous())
    state = run._replay_segment(0, 1)[0]
    lam = torch.tensor(np.random.default_rng(3).standard_normal((4, mesh.n_real)), device="cuda")
    quads = run._adjoint(rec, state, lam)
    one = run._adjoint(rec, state[:3] + (None,), lam)
    assert bool(torch.isfinite(quads).all())
    # the same operations in the same order; the recomputed limiter values may differ in the last place
    assert float((quads - one).abs().max()) <= 1e-13 * float(one.abs().max())
