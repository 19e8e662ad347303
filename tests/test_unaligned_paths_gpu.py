"""Large forwards with unaligned operands by the plan's path: by default on CUDA
cores, whose FP16 result is the FP32 one rounded; on the tensor cores only for a
plan that asks for them (path 2), also with infinities and NaN in B.

Tolerance there, elementwise: |error| <= n_r 2^-23 (|A| |B|)[r, n] plus 2^-11
|ref| + 2^-24 for the FP16 output, and one FP32 rounding more for beta (2^-23 of
the result)."""
import numpy as np
import pytest

from test_unaligned_gpu import case

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import tca_spmm  # noqa: E402

SHAPES = [(700, 1100, 99, 0.5), (513, 770, 264, 0.4), (900, 400, 513, 0.3)]


def operand(Bh, cuda):
    """B on the GPU, its rows at odd offsets (N may be a multiple of 8)."""
    wide = torch.zeros((Bh.shape[0], Bh.shape[1] + 3), dtype=torch.float16, device=cuda)
    wide[:, 1:-2] = torch.from_numpy(Bh).to(cuda)
    return wide[:, 1:-2]


@pytest.mark.parametrize("M,K,N,density", SHAPES)
def test_default_rounds_the_fp32_sums(cuda, M, K, N, density):
    dev, Bh, _, _ = case(M, K, N, density, cuda, M)
    plan, B = tca_spmm.Plan(*dev, K), operand(Bh, cuda)
    assert plan.info()["n_tc_windows"] > 0 and dev[1].numel() * N >= 2 ** 25
    half, full = plan.spmm(B, out_dtype=torch.float16), plan.spmm(B, out_dtype=torch.float32)
    assert torch.equal(half, full.half())


@pytest.mark.parametrize("M,K,N,density", SHAPES)
@pytest.mark.parametrize("bad", [None, float("inf"), float("nan")])
def test_tensor_core_plan(cuda, M, K, N, density, bad):
    dev, Bh, A, n_r = case(M, K, N, density, cuda, M + 1)
    b64 = Bh.astype(np.float64)
    ref, mag = A @ b64, np.abs(A) @ np.abs(b64)
    clean = np.ones((M, N), dtype=bool)
    if bad is not None:
        Bh[17, 40] = bad
        clean[:, 40] = A[:, 17] == 0
    plan = tca_spmm.Plan(*dev, K, path="tensor_core")
    C = torch.full((M, N), 0.5, dtype=torch.float16, device=cuda)
    plan.spmm(operand(Bh, cuda), out=C, alpha=2.0, beta=0.5, keep_empty_rows=True)
    plan.status()
    got, want = C.cpu().numpy().astype(np.float64), np.where(n_r > 0, 2 * ref + 0.25, 0.5)
    tol = 2 * n_r * 2.0 ** -23 * mag + 2.0 ** -23 * np.abs(want) + 2.0 ** -11 * np.abs(want) + 2.0 ** -24
    assert np.all(np.abs(got - want)[clean] <= tol[clean])
    assert not np.isfinite(got[~clean]).any()
