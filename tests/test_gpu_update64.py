"""The FP64 step's last kernel (segmented sums, recovery, time step, phd_f64.cu) and the
generator velocities in its first one, against the oracle (FP64, 1e-12): around the edges of
a block, with negative masses reported, with a cell whose generator sits on its centroid, and
where quotients fall back on the plain operations (totals beyond the seeds' window)."""
import numpy as np
import pytest

import oracle as O
import phd_code_gb300 as pkg
from _util import assert_parity, lattice_mesh, smooth_state
from phd_code_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("recon", ["linear", "constant"])
@pytest.mark.parametrize("side,boundary,scale", [(4, "periodic", 1.0), (9, "reflective", 1.0), (12, "periodic", 1e90),
                                                 (12, "reflective", 1e-130), (31, "periodic", 1.0)])
def test_moving_steps_match_oracle(side, boundary, scale, recon):
    mesh = lattice_mesh(side, boundary, seed=9)
    mesh.dcom[:, 0] = 0.0                       # a generator on its centroid (and its images)
    mesh.dcom[:, mesh.map == 0] = 0.0
    mesh.dcom[:, 1] *= 10.0                     # one far off it, one on the edge of steering
    mesh.dcom[:, mesh.map == 1] = mesh.dcom[:, [1]]
    prim = smooth_state(mesh)
    prim[0] *= scale                            # density and pressure together: the same speeds
    prim[3] *= scale
    st = pkg.FluxStepper(mesh, prim, gamma=1.4, solver="hll", moving=True, reconstruction=recon)
    ost = O.OracleStepper(mesh, gamma=1.4, solver="hll", moving=True, linear=recon == "linear")
    p, c = prim.copy(), O.cons_from_prim(mesh, prim, 1.4)
    for _ in range(2):
        ost.step(O.time_step(mesh, p, 1.4, 0.5, True), p, c)
        st.step(1)
    st.check_status()
    assert_parity(st.cons_host(), c)
    assert_parity(st.prim_host(), p)
    assert abs(st.read_clock().dt - O.time_step(mesh, p, 1.4, 0.5, True)) <= 1e-12 * st.read_clock().dt


def test_negative_mass_and_energy_are_reported():
    mesh = lattice_mesh(8, "periodic", seed=9)
    st = pkg.FluxStepper(mesh, smooth_state(mesh), gamma=1.4, solver="hllc")
    st.clock.set(dt=50.0)
    st.step(1)
    assert st.read_clock().status & (L.STATUS_NEG_MASS | L.STATUS_NEG_ENERGY)
