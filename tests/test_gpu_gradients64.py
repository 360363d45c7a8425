"""The FP64 gradient kernel works on blocks of 32 rows, face by face (phd_f64.cu): the
oracle's gradients (FP64, 1e-12) at sizes around the block's edges, with both limiters and
boundaries, and where a block takes its plain path -- a cell with more faces than the
block's shared lists hold, values outside the seeds' exponent window -- and the taped
gradients equal to the untaped ones bit for bit."""
import numpy as np
import pytest
import torch

import oracle as O
import phd_code_gb300 as pkg
from _util import assert_parity, lattice_mesh, smooth_state
from phd_code_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def device_gradients(mesh, prim, limiter, taped=False):
    dm = pkg.DeviceMesh(mesh)
    n = mesh.n_cells
    p = torch.as_tensor(np.ascontiguousarray(prim)).cuda()
    g = torch.zeros((8, n), dtype=torch.float64, device="cuda")
    clk = pkg.DeviceClock()
    lim = L.LIMITER_AREPO if limiter == "arepo" else L.LIMITER_TESS
    if taped:
        tf = torch.zeros((L.GRAD_TAPE_F64_ROWS, n), dtype=torch.float64, device="cuda")
        ti = torch.zeros((L.GRAD_TAPE_I32_ROWS, n), dtype=torch.int32, device="cuda")
        L.check(L.lib().phd_gradients_f64_taped(dm.ref, L.ptr(p), lim, L.ptr(g), L.ptr(tf), L.ptr(ti), clk.ptr,
                                                L.stream_handle()), "taped")
        clk.check_status()
        return g.cpu().numpy(), tf.cpu().numpy(), ti.cpu().numpy()
    L.check(L.lib().phd_gradients_f64(dm.ref, L.ptr(p), lim, L.ptr(g), clk.ptr, L.stream_handle()), "gradients")
    clk.check_status()
    return g.cpu().numpy()


def ring_mesh():
    """A cell in the middle of a ring of 300: its list overflows a block's shared lists."""
    a = np.linspace(0.0, 2.0 * np.pi, 300, endpoint=False)
    ring = np.stack([0.5 + 0.3 * np.cos(a), 0.5 + 0.3 * np.sin(a)])
    rng = np.random.default_rng(4)
    out = rng.uniform(0.02, 0.98, (2, 400))
    out = out[:, np.hypot(out[0] - 0.5, out[1] - 0.5) > 0.33]
    return pkg.meshgen.build_mesh(np.concatenate([[[0.5], [0.5]], ring, out], axis=1), "periodic")[0]


@pytest.mark.parametrize("limiter", ["arepo", "tess"])
@pytest.mark.parametrize("kind", ["4 periodic", "5 reflective", "6 periodic", "8 reflective", "23 periodic",
                                  "40 reflective", "ring", "huge", "tiny"])
def test_gradients_match_oracle(kind, limiter):
    if kind == "ring":
        mesh = ring_mesh()
        assert np.diff(mesh.nbr_ptr).max() > 256
    elif kind in ("huge", "tiny"):
        mesh = lattice_mesh(12, "periodic", seed=5)
    else:
        mesh = lattice_mesh(int(kind.split()[0]), kind.split()[1], seed=5)
    prim = smooth_state(mesh)
    if kind == "huge":
        prim[:, mesh.x[0] > 0.5] *= 2.0 ** 600
        prim = pkg.meshgen.fill_ghosts(mesh, prim)
    elif kind == "tiny":
        prim *= 2.0 ** -560
    want, status = O.gradients(mesh, prim, 0 if limiter == "arepo" else 1)
    assert status == 0
    got = device_gradients(mesh, prim, limiter)
    assert_parity(got, want)
    g, tf, ti = device_gradients(mesh, prim, limiter, taped=True)
    assert np.array_equal(g, got)
    # the record reproduces the limited gradient, and its entries lie in the cell's list
    nr = mesh.n_real
    assert np.array_equal(np.repeat(tf[8:12, :nr], 2, axis=0) * tf[:8, :nr], g[:, :nr])
    e = ti[:12, :nr]
    assert np.all((e < 0) | ((e >= mesh.nbr_ptr[:nr]) & (e < mesh.nbr_ptr[1:nr + 1])))


@pytest.mark.parametrize("scale", [2.0 ** -300, 1.0, 2.0 ** 200])
@pytest.mark.parametrize("slope", [(1.0, 1.0), (1.0, -1.0), (1.0, 0.0), (0.0, 0.0), (1.0, 2.0 ** -40)])
def test_largest_change_among_equals(slope, scale):
    """The limiter's face where several are equal or nearly so: regular lattices, where the
    separations repeat up to their rounding, with slopes along the axes and the diagonals."""
    mesh, _ = pkg.meshgen.build_mesh(pkg.meshgen.jittered_lattice(9, jitter=0.0, seed=1), "reflective")
    wave = slope[0] * mesh.x[0] + slope[1] * mesh.x[1]
    bump = np.where((mesh.x[0] > 0.4) & (mesh.x[1] > 0.4), 1.0, 0.0)
    prim = pkg.meshgen.fill_ghosts(mesh, np.stack([3.0 + wave, wave, bump, 3.0 + bump + wave]) * scale)
    want, status = O.gradients(mesh, prim, 0)
    assert status == 0
    got = device_gradients(mesh, prim, "arepo")
    assert_parity(got, want)
