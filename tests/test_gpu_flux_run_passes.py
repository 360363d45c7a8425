"""Passes through one recorded run: each backward pass belongs to its own forward pass, whatever ran
in between, and a forward pass that no gradient can follow records nothing for one."""
import gc

import pytest
import torch

import phd_code_gb300 as pkg
from phd_code_gb300.adjoint import FluxRun, FluxRunRecord, StepRecord

pytestmark = pytest.mark.gpu


def _run(steps, checkpoint):
    mesh, prim, _ = pkg.problems.gaussian_bump(16, background=False)
    st = pkg.FluxStepper(mesh, prim, gamma=1.4, moving=True)
    recs = []
    for _ in range(steps):
        dt = st.read_clock().dt
        st.step(1)
        recs.append(StepRecord(st.dmesh, st.face_w.clone(), dt))
    return FluxRunRecord(recs, gamma=1.4, checkpoint=checkpoint), torch.tensor(prim[:, :mesh.n_real], device="cuda")


@pytest.mark.parametrize("steps, checkpoint", [(1, 20), (5, 20), (7, 3), (5, 1)])
def test_a_gradient_is_of_its_own_forward_pass(steps, checkpoint):
    run, p0 = _run(steps, checkpoint)
    lam = torch.linspace(-1.0, 1.0, run.n_real, dtype=torch.float64, device="cuda")
    states = [p0, p0 * torch.tensor([[1.3], [1.0], [1.0], [0.8]], dtype=torch.float64, device="cuda")]

    def alone(x):
        p = x.clone().requires_grad_(True)
        FluxRun.apply(p, run).backward(lam)
        return p.grad

    want = [alone(x) for x in states]
    assert not torch.equal(*want)
    ps = [x.clone().requires_grad_(True) for x in states]
    outs = [FluxRun.apply(p, run) for p in ps]
    with torch.no_grad():
        FluxRun.apply(states[1], run)
    for out, p, g in zip(outs, ps, want):              # the first forward's backward first
        out.backward(lam, retain_graph=True)
        assert torch.equal(p.grad, g)
    ps[0].grad = None
    outs[0].backward(lam)                              # and once more, the second's in between
    assert torch.equal(ps[0].grad, want[0])


def test_a_dropped_graph_takes_its_record_with_it():
    run, p0 = _run(5, 20)
    out = FluxRun.apply(p0.clone().requires_grad_(True), run)
    assert run._tail is not None
    del out
    gc.collect()
    assert run._tail is None


def test_no_record_without_a_gradient(monkeypatch):
    run, p0 = _run(5, 20)
    taped = []
    step = FluxRunRecord._step
    monkeypatch.setattr(FluxRunRecord, "_step",
                        lambda self, k, *a, **kw: (taped.append(len(a) > 4 and a[4] is not None), step(self, k, *a, **kw))[1])
    p = p0.clone().requires_grad_(True)
    with torch.no_grad():
        rho = FluxRun.apply(p, run)
    assert run._tail is None and not any(taped)
    assert torch.equal(rho, FluxRun.apply(p0, run)) and not any(taped)
    out = FluxRun.apply(p, run)
    assert torch.equal(out.detach(), rho) and any(taped) and run._tail is not None
