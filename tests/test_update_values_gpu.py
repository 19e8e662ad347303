"""New values for a plan: the one-launch update against a plan built from those
values, array by array and bit for bit, and its transpose; chunks from a few
entries to full (8192), entry counts off the block sizes. And gradients when
another forward replaced the values in between."""
import numpy as np
import pytest

from tca_spmm import gen

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import tca_spmm  # noqa: E402
from tca_spmm import autograd  # noqa: E402


@pytest.mark.parametrize("M,K,density", [(1, 70, 0.5), (130, 64, 1.0), (700, 300, 0.3), (513, 400, 0.05), (900, 333, 0.008)])
@pytest.mark.parametrize("transpose", [False, True])
def test_update_matches_fresh_plan(cuda, M, K, density, transpose):
    rng = np.random.default_rng(M + K)
    c = gen.small(rng, M, K, 72, density, empty_rows=0.1)
    v2 = rng.standard_normal(c["col"].size).astype(np.float16)
    rp, ci, v, B = (torch.from_numpy(c[k].copy()).to(cuda) for k in ("row_ptr", "col", "vals", "B"))
    plan = tca_spmm.Plan(rp, ci, v, K)
    if transpose:
        plan.build_transpose()
    n0 = plan.values_version()
    new = torch.from_numpy(v2).to(cuda)
    plan.update_values(new)
    assert c["col"].size == 0 or plan.values_version() == n0 + 1
    fresh = tca_spmm.Plan(rp, ci, new, K)
    for which in (tca_spmm.ARR_P_VAL, tca_spmm.ARR_TILE_ENTRIES, tca_spmm.ARR_TILE_IMAGES):
        assert np.array_equal(plan.export(which), fresh.export(which))
    dY = torch.randn((M, 72), device=cuda).half()
    assert torch.equal(plan.spmm_t(dY), fresh.spmm_t(dY))
    assert torch.equal(plan.spmm(B), fresh.spmm(B))


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_backward_after_other_values(cuda, dtype):
    rng = np.random.default_rng(5)
    c = gen.small(rng, 300, 200, 64, 0.15)
    rp, ci, v, B = (torch.from_numpy(c[k].copy()).to(cuda) for k in ("row_ptr", "col", "vals", "B"))
    plan = tca_spmm.Plan(rp, ci, v, 200)
    dY = torch.randn((300, 64), device=cuda)
    grads = []
    for other in (False, True):
        a, b = v.to(dtype).requires_grad_(), B.to(dtype).requires_grad_()
        Y = autograd.spmm(plan, a, b)
        if other:  # another forward on the plan between this one and its backward
            autograd.spmm(plan, -2 * a.detach(), b.detach())
        grads.append(torch.autograd.grad(Y, (a, b), dY))
    for x, y in zip(*grads):
        assert x.dtype == dtype and torch.equal(x, y)


def test_first_cuda_call_of_a_thread(cuda):
    """A backward pass can be the first CUDA call of its host thread (as
    autograd's is): the tensor maps are encoded without a current context."""
    import threading
    rng = np.random.default_rng(6)
    c = gen.small(rng, 300, 200, 64, 0.15)
    rp, ci, v, B = (torch.from_numpy(c[k].copy()).to(cuda) for k in ("row_ptr", "col", "vals", "B"))
    plan = tca_spmm.Plan(rp, ci, v, 200)
    dY = torch.randn((300, 64), device=cuda).half()
    want, got = plan.sddmm(dY, B), torch.empty(c["col"].size, device=cuda)
    Y, Y2 = plan.spmm(B), torch.empty((300, 64), dtype=torch.float16, device=cuda)
    torch.cuda.synchronize()
    errors = []

    def call(f):
        try:
            f()
        except Exception as e:
            errors.append(e)

    stream = torch.cuda.current_stream()
    for f in (lambda: plan.sddmm(dY, B, out=got, stream=stream), lambda: plan.spmm(B, out=Y2, stream=stream)):
        t = threading.Thread(target=call, args=(f,))
        t.start()
        t.join()
    torch.cuda.synchronize()
    assert not errors and torch.equal(got, want) and torch.equal(Y, Y2)
