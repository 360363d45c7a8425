"""The time step of a fused FP64 step where p / rho leaves FP32's normal range (its cells are
compared in FP32 first): the plain reduction over the same primitives, bit for bit."""
import numpy as np
import pytest
import torch

import phd_code_gb300 as pkg
from _util import lattice_mesh, smooth_state
from phd_code_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("boost", [True, False])
@pytest.mark.parametrize("log2_rho, log2_p", [(0, 0), (0, -99), (40, -60), (60, -66), (68, -70), (74, -69), (76, -69),
                                              (90, -90), (-90, 90), (-30, -150), (120, 3)])
def test_smallest_candidate_is_found(log2_rho, log2_p, boost):
    mesh = lattice_mesh(31, "periodic", seed=9)
    prim = smooth_state(mesh)
    prim[0] *= 2.0 ** log2_rho
    prim[1:3] *= 2.0 ** ((log2_p - log2_rho) // 2)        # Mach numbers as they were
    prim[3] *= 2.0 ** log2_p
    st = pkg.FluxStepper(mesh, prim, gamma=1.4, solver="hll", boost=boost, moving=False)
    st.clock.set(dt=0.0)                        # the state stays as it is
    st.step(1)
    st.check_status()
    clk = pkg.DeviceClock()
    L.check(L.lib().phd_time_step_f64(st.dmesh.ref, L.ptr(st.prim), 1.4, 0.5, int(boost), 0, clk.ptr,
                                      L.stream_handle()), "phd_time_step_f64")
    assert 0.0 < clk.read().dt < np.inf
    assert st.read_clock().dt == clk.read().dt
