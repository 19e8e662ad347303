"""Large forwards with unaligned operands take scratch memory: one thread's must
not disturb a graph capture that another thread has under way, nor be refused
because of it."""
import threading

import numpy as np
import pytest

from tca_spmm import gen

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import tca_spmm  # noqa: E402


@pytest.mark.parametrize("planned", [True, False])
@pytest.mark.parametrize("out", ["f16", "f32"])
def test_forward_beside_a_capture(cuda, planned, out):
    c = gen.small(np.random.default_rng(2), 1500, 1000, 203, 0.15)  # nnz * N = 4.6e7
    rp, ci, v, B = (torch.from_numpy(c[k]).to(cuda) for k in ("row_ptr", "col", "vals", "B"))
    plan = tca_spmm.Plan(rp, ci, v, 1000)
    stream, other = torch.cuda.Stream(), torch.cuda.Stream()
    dt = torch.float16 if out == "f16" else torch.float32
    got, want = (torch.empty((1500, 203), dtype=dt, device=cuda) for _ in range(2))

    def forward(C):
        if planned:
            plan.spmm(B, out=C, stream=stream)
        else:
            tca_spmm.spmm_csr(rp, ci, v, B, out=C, stream=stream)

    x, errors = torch.zeros(8, device=cuda), []
    torch.cuda.synchronize()
    forward(want)
    torch.cuda.synchronize()

    def call():
        try:
            forward(got)
        except Exception as e:
            errors.append(e)

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=other):
        x.add_(1)
        t = threading.Thread(target=call)
        t.start()
        t.join()
        x.add_(1)
    graph.replay()
    torch.cuda.synchronize()
    assert not errors and torch.equal(got, want) and torch.all(x == 2)
