"""A solver number that phd_step_f64 has no name for runs HLL, as it always has: the same bits, in
one call and in several."""
import numpy as np
import pytest

import phd_code_gb300 as pkg
from _util import lattice_mesh, smooth_state
from phd_code_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("boost", [True, False])
@pytest.mark.parametrize("number", [-1, 3, 7])
def test_runs_hll(number, boost):
    mesh = lattice_mesh(9, "reflective", seed=2)
    assert number not in (L.HLL, L.HLLC, L.EXACT)
    a = pkg.FluxStepper(mesh, smooth_state(mesh), gamma=1.4, solver="hll", boost=boost)
    b = pkg.FluxStepper(mesh, smooth_state(mesh), gamma=1.4, solver=number, boost=boost)
    for n in (1, 2):
        a.step(n)
        b.step(n)
        a.check_status()
        b.check_status()
        assert np.array_equal(a.cons_host(), b.cons_host()) and np.array_equal(a.prim_host(), b.prim_host())
        assert a.read_clock().dt == b.read_clock().dt
