"""The gradients of the differentiable form are tensors of their own, as a
caller of torch.autograd may expect: none shares memory or a version with
another, each may be written to, with and without create_graph."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from openmmcustomgbintegralforce_gb300.autograd import GBEnergy  # noqa: E402
from openmmcustomgbintegralforce_gb300.globule import make_globule  # noqa: E402
from openmmcustomgbintegralforce_gb300.spec import GBModel  # noqa: E402

pytestmark = pytest.mark.gpu

DTYPES = [("float64",) * 4, ("float32",) * 4, ("float32", "float64", "float32", "float64")]


@pytest.fixture(params=DTYPES, ids=["double", "single", "mixed"])
def case(request):
    g = make_globule(300, seed=6)
    m = GBModel.charmm_gbsw()
    values = [g.positions, g.charge, g.radius, np.array([m.alpha0, m.alpha1])]
    leaves = [torch.tensor(v, dtype=getattr(torch, d), device="cuda:0", requires_grad=True)
              for v, d in zip(values, request.param)]
    return GBEnergy(m, g.n), leaves


def test_no_gradient_holds_another_s_memory(case):
    mod, leaves = case
    grads = torch.autograd.grad(mod(*leaves), leaves)
    assert len({t.untyped_storage().data_ptr() for t in grads}) == 4
    assert all(t.untyped_storage().nbytes() == t.numel() * t.element_size() for t in grads)
    assert all(t.dtype == p.dtype and t.shape == p.shape and t.is_contiguous() for t, p in zip(grads, leaves))


@pytest.mark.parametrize("kept", range(4))
def test_writing_to_one_gradient_leaves_the_others(case, kept):
    mod, leaves = case
    grads = torch.autograd.grad(mod(*leaves), leaves)
    w = torch.ones_like(grads[kept]).requires_grad_()
    loss = (w * grads[kept]).sum()  # saves the gradient for its own backward
    want = grads[kept].clone()
    for k, t in enumerate(grads):
        if k != kept:
            t.zero_()
    loss.backward()
    assert torch.equal(w.grad, want)


def test_gradients_can_be_written_to_in_a_graph(case):
    mod, leaves = case
    plain = torch.autograd.grad(mod(*leaves), leaves)
    s = torch.tensor(2.0, dtype=torch.float64, device="cuda:0", requires_grad=True)
    # as a graph's own tensors: each scaled in place, then differentiated
    grads = torch.autograd.grad(s * mod(*leaves), leaves, create_graph=True)
    total = sum(t.mul_(3.0).double().sum() for t in grads)
    (ds,) = torch.autograd.grad(total, s)
    want = 3.0 * sum(t.double().sum() for t in plain)
    # s scales every gradient: its own is their sum, to single precision's rounding of each
    scale = 3.0 * sum(t.double().abs().sum() for t in plain)
    assert abs(float(ds - want)) < 4e-7 * float(scale)
    # and without a graph, by a factor that asks for one
    for t in plain:
        w = torch.ones_like(t).requires_grad_()
        t.mul_(w).sum().backward()
        assert w.grad is not None
