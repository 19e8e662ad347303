"""SDDMM work units at their edges: chunk groups of 8, of fewer (few n steps)
and a ragged last group; halves of consecutive chunks (one box) and not
(condensed columns, a window that skips blocks of K); windows of consecutive
rows (one box) and permuted ones (gathered); one part and several with ragged
entry ranges; N not a multiple of the 64-wide step.

Tolerance, elementwise: |error| <= N 2^-23 sum_n |dY| |B| (exact products
accumulated in FP32 in any order, FP32 sums of the parts), plus 2^-11 |ref| +
2^-24 for FP16 output."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import tca_spmm  # noqa: E402


def pattern(kind, M, K, rng):
    mask = rng.random((M, K)) < 0.12
    if kind == "even":  # equal rows: windows of consecutive rows
        mask = np.zeros((M, K), bool)
        for r in range(M):
            mask[r, rng.choice(K, K // 8, replace=False)] = True
    elif kind == "skip":  # blocks of K that a window does not touch: runs broken
        mask[:, 64:128] = False
        mask[: M // 2, 256:320] = False
    elif kind == "condensed":
        keep = np.zeros(K, bool)
        keep[rng.choice(K, K // 7, replace=False)] = True
        mask = (rng.random((M, K)) < 0.5) & keep
    return mask


@pytest.mark.parametrize("kind", ["even", "binomial", "skip", "condensed"])
@pytest.mark.parametrize("M,K,N", [(128, 64, 64), (300, 512, 64), (257, 832, 200), (640, 600, 1024), (130, 1100, 72)])
@pytest.mark.parametrize("out", ["f16", "f32"])
def test_sddmm_units(cuda, kind, M, K, N, out):
    rng = np.random.default_rng(M + K + N)
    mask = pattern(kind, M, K, rng)
    rows, cols = np.nonzero(mask)
    rp = np.concatenate([[0], np.cumsum(mask.sum(1))]).astype(np.int32)
    vals = rng.standard_normal(cols.size).astype(np.float16)
    dY = rng.standard_normal((M, N)).astype(np.float16)
    B = rng.standard_normal((K, N)).astype(np.float16)
    t = [torch.from_numpy(x).to(cuda) for x in (rp, cols.astype(np.int32), vals, dY, B)]
    plan = tca_spmm.Plan(*t[:3], K, path="tensor_core")
    got = plan.sddmm(t[3], t[4], out_dtype=torch.float16 if out == "f16" else torch.float32, alpha=0.5)
    plan.status()
    y, b = dY.astype(np.float64), B.astype(np.float64)
    ref = 0.5 * (y @ b.T)[rows, cols]
    mag = 0.5 * (np.abs(y) @ np.abs(b).T)[rows, cols]
    tol = N * 2.0 ** -23 * mag + (2.0 ** -11 * np.abs(ref) + 2.0 ** -24 if out == "f16" else 0)
    assert np.all(np.abs(got.cpu().numpy().astype(np.float64) - ref) <= tol)
