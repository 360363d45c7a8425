"""A stepper's first hand-over looks the current stream up a few times, not once for each of the
events that it makes (up to 5 us each; the first pass on a new stepper of 512 x 512 cells took 491 us, against 448)."""
import pytest
import torch

import phd_code_gb300 as pkg
from _util import lattice_mesh, smooth_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("compact", [True, False])
def test_stream_is_looked_up_once(compact, monkeypatch):
    mesh = lattice_mesh(8, "periodic", seed=1)
    st = pkg.FluxStepper(mesh, smooth_state(mesh), precision="fp32")
    pinned = st.dmesh.pinned_host_compact(mesh) if compact else st.dmesh.pinned_host()
    looked = []
    main = pkg.FluxStepper._main_stream
    monkeypatch.setattr(pkg.FluxStepper, "_main_stream", lambda self: (looked.append(1), main(self))[1])
    st.load_mesh(pinned)
    torch.cuda.synchronize()
    assert len(looked) <= 3
    del looked[:]
    st.load_mesh(pinned)                        # the second has no events left to make
    torch.cuda.synchronize()
    assert len(looked) <= 1
