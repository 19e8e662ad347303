"""Gradients where a CUDA graph replaces the plan's values between a forward and
its backward, or runs the backward: each backward uses the values of its own
forward, as in a run without graphs (compared bit for bit)."""
import numpy as np
import pytest

from tca_spmm import gen

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import tca_spmm  # noqa: E402
from tca_spmm import autograd  # noqa: E402


@pytest.fixture
def problem(cuda):
    c = gen.small(np.random.default_rng(8), 300, 200, 64, 0.15)
    rp, ci, v, B = (torch.from_numpy(c[k].copy()).to(cuda) for k in ("row_ptr", "col", "vals", "B"))
    plan = tca_spmm.Plan(rp, ci, v, 200)
    plan.build_transpose()
    dY = torch.randn((300, 64), device=cuda)
    a, b = v.requires_grad_(), B.requires_grad_()
    want = torch.autograd.grad(autograd.spmm(plan, a, b), (a, b), dY)
    torch.cuda.synchronize()
    return plan, a, b, dY, want


def test_replayed_forward_between(problem):
    plan, a, b, dY, want = problem
    other = (-2 * a).detach()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        autograd.spmm(plan, other, b.detach())
    for _ in range(2):
        Y = autograd.spmm(plan, a, b)
        graph.replay()
        got = torch.autograd.grad(Y, (a, b), dY)
        assert all(torch.equal(x, y) for x, y in zip(got, want))


def test_forward_captured_before_the_plan_is_used_eagerly(problem):
    plan, a, b, dY, want = problem
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        Y = autograd.spmm(plan, a, b)
    graph.replay()
    autograd.spmm(plan, (3 * a).detach(), b.detach())
    torch.cuda.synchronize()
    got = torch.autograd.grad(Y, (a, b), dY)
    assert all(torch.equal(x, y) for x, y in zip(got, want))


def test_captured_backward(problem):
    plan, a, b, dY, want = problem
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        Y = autograd.spmm(plan, a, b)
        torch.autograd.grad(Y, (a, b), dY, retain_graph=True)  # warm-up
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        got = torch.autograd.grad(Y, (a, b), dY)
    autograd.spmm(plan, (5 * a).detach(), b.detach())
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(x, y) for x, y in zip(got, want))
