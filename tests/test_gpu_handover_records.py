"""``handover_records`` may change between compact hand-overs of equal counts: the records that a
step reads are those of the mesh it runs on, so the steps equal, bit for bit, those of a stepper
that never reads any."""
import numpy as np
import pytest
import torch

import phd_code_gb300 as pkg
from _util import lattice_mesh, smooth_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [(False, True), (True, False, True), (False, True, False, True), (True, True, False)])
@pytest.mark.parametrize("limiter", ["arepo", "tess"])
def test_records_follow_the_attribute(flags, limiter):
    mesh = lattice_mesh(14, "periodic", seed=3)
    real = mesh.x[:, :mesh.n_real]
    meshes = []
    for k in range(len(flags)):               # generators moved too little to change a neighbour
        moved = real + 1e-5 * (k + 1) * np.sin(7.0 * real[::-1])
        m, order = pkg.meshgen.build_mesh(moved, "periodic", hilbert=False)
        assert (m.n_cells, m.n_faces) == (mesh.n_cells, mesh.n_faces)
        meshes.append(m)
    kw = dict(gamma=1.4, solver="hllc", moving=True, precision="fp32", limiter=limiter)
    a = pkg.FluxStepper(mesh, smooth_state(mesh), **kw)
    b = pkg.FluxStepper(mesh, smooth_state(mesh), **kw)
    for m, flag in zip(meshes, flags):
        a.handover_records = flag
        a.load_mesh(a.dmesh.pinned_host_compact(m))
        b.load_mesh(b.dmesh.pinned_host_compact(m))
        assert a.records == flag and (a.geo.entry_rec is not None) == flag
        assert not b.records and b.geo.entry_rec is None
        a.step(1)
        b.step(1)
        torch.cuda.synchronize()
        assert torch.equal(a.cellrec, b.cellrec)
        assert np.array_equal(a.cons_host(), b.cons_host())


@pytest.mark.parametrize("compact", [True, False])
def test_a_captured_graph_reads_the_new_meshs_records(compact):
    """A graph outlives a hand-over of equal counts; its steps read records, and a replay builds those
    that the hand-over left unwritten."""
    mesh = lattice_mesh(14, "periodic", seed=3)
    real = mesh.x[:, :mesh.n_real]
    other, _ = pkg.meshgen.build_mesh(real + 1e-5 * np.sin(7.0 * real[::-1]), "periodic", hilbert=False)
    assert (other.n_cells, other.n_faces) == (mesh.n_cells, mesh.n_faces)
    a, b = (pkg.FluxStepper(mesh, smooth_state(mesh), gamma=1.4, moving=True, precision="fp32") for _ in range(2))
    a.capture(2)
    for st in (a, b):
        st.load_mesh(st.dmesh.pinned_host_compact(other) if compact else st.dmesh.pinned_host(other))
    assert not a.records
    for _ in range(2):
        a.replay()
        b.step(2)
        torch.cuda.synchronize()
        assert a.records and np.array_equal(a.cons_host(), b.cons_host())
