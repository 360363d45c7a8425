"""The FP32 step's kernels load their mesh rows ahead of the wait for the previous kernel
where the grid covers the mesh, and in place where their threads loop over it: the same
bits, ghosts, short last blocks and a mesh handed over just before the step included."""
import numpy as np
import pytest

import phd_code_gb300 as pkg
import phd_code_gb300._lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [5, 16, 33])
@pytest.mark.parametrize("solver, limiter, reconstruction, moving", [
    ("hllc", "arepo", "linear", True), ("hll", "tess", "linear", False),
    ("exact", "arepo", "constant", True), ("hllc", "arepo", "constant", False)])
def test_covering_and_looping_grids_agree(side, solver, limiter, reconstruction, moving):
    mesh, prim, cfg = pkg.problems.shock_tube(side)
    cons = []
    for launch in (None, L.PhdLaunch(32, 32, 32, 2, 2, 2, 1, 1, 1), L.PhdLaunch(64, 64, 64, 0, 0, 0, 2, 2, 2)):
        st = pkg.FluxStepper(mesh, prim, gamma=cfg["gamma"], solver=solver, limiter=limiter, reconstruction=reconstruction,
                             moving=moving, precision="fp32")
        st.launch = launch
        st.step(2)
        st.load_mesh(st.dmesh.pinned_host(mesh))
        st.step(3)
        st.check_status()
        cons.append(st.cons_host())
    assert np.isfinite(cons[0]).all()
    assert np.array_equal(cons[0], cons[1]) and np.array_equal(cons[0], cons[2])
