"""The autograd wrappers of the differentiable costs: the gradient is formed in the forward pass only where q
needs one, and what autograd accepted and refused stays so."""
import numpy as np
import pytest

from plainmp_gb300 import diff, scenes
from plainmp_gb300 import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def setup():
    _, cst, _ = scenes.make_constraint(W.chain7_robot(), W.chain7_scene())
    rng = np.random.default_rng(2)
    q = torch.tensor(W.chain7_configs(70, seed=4), dtype=torch.float32, device="cuda")
    t = np.concatenate([rng.normal(0, 0.3, (70, 3)), np.tile([0, 0, 0, 1.0], (70, 1))], axis=1)
    off = torch.tensor([0, 1, 30, 70], device="cuda")
    return cst, q, torch.tensor(t, dtype=torch.float32, device="cuda"), off


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_gradients_match_the_direct_call(setup, dtype):
    cst, q, t, off = setup
    w = torch.linspace(-1.0, 2.0, 70, device="cuda")
    x = q.to(dtype).requires_grad_(True)
    cost = diff.ik_cost(cst, x, t, "link7")
    ref, g = diff.ik_cost_grad(cst, q, t, "link7")
    assert torch.equal(cost, ref)
    (dx,) = torch.autograd.grad((w * cost).sum(), x, retain_graph=True)
    assert dx.dtype is dtype and torch.equal(dx, (w[:, None] * g).to(dtype))
    (again,) = torch.autograd.grad((w * cost).sum(), x)
    assert torch.equal(again, dx)
    wt = torch.tensor([1.0, -0.5, 2.0], device="cuda")
    tc = diff.trajectory_cost(cst, x, off)
    tref, tg = diff.traj_cost_grad(cst, q, off)
    assert torch.equal(tc, tref)
    (dx,) = torch.autograd.grad((wt * tc).sum(), x)
    assert torch.equal(dx, (torch.repeat_interleave(wt, off.diff())[:, None] * tg).to(dtype))


def test_no_gradient_wanted(setup):
    cst, q, t, off = setup
    ref = diff.ik_cost_grad(cst, q, t, "link7", want_grad=False)
    assert torch.equal(diff.ik_cost(cst, q, t, "link7"), ref)
    with torch.no_grad():
        assert torch.equal(diff.ik_cost(cst, q.clone().requires_grad_(True), t, "link7"), ref)
    tt = t.clone().requires_grad_(True)  # only the target asks for one: none comes back
    assert torch.autograd.grad(diff.ik_cost(cst, q, tt, "link7").sum(), tt, allow_unused=True) == (None,)


def test_change_in_place_is_refused(setup):
    cst, q, t, off = setup
    for make in (lambda x: diff.ik_cost(cst, x, t, "link7"), lambda x: diff.trajectory_cost(cst, x, off)):
        x = q.clone().requires_grad_(True)
        cost = make(x)
        with torch.no_grad():
            x += 1.0
        with pytest.raises(RuntimeError, match="modified by an inplace"):
            cost.sum().backward()


@pytest.mark.parametrize("mode", [torch.no_grad, torch.inference_mode])
def test_no_gradient_is_formed_where_none_is_recorded(setup, mode):
    """A leaf that asks for gradients, in a call that records none: the cost alone, by the memory it takes."""
    cst, q, t, off = setup
    x = q.repeat(3000, 1).requires_grad_(True)  # its gradient: 5.9 MB; the cost 0.8 MB
    tt = t.repeat(3000, 1)
    offs = torch.arange(0, len(x) + 1, 70, device="cuda")
    for call in (lambda: diff.ik_cost(cst, x, tt, "link7"), lambda: diff.trajectory_cost(cst, x, offs)):
        with mode():
            call()
            torch.cuda.synchronize()
            before = torch.cuda.memory_allocated()
            torch.cuda.reset_peak_memory_stats()
            cost = call()
            assert torch.cuda.max_memory_allocated() - before < 4 * x.numel()
            assert not cost.requires_grad
