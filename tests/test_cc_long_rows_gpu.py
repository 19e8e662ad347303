"""CUDA-core windows with few, long rows (a ragged last window): the rows kernel
over part of a plan's rows (FP16), the stream kernel with N cut into slices
(E4M3, and FP16 with an explicit cc_cols); with and without tensor-core windows
before them, rows without nonzeros, alpha and beta, several jobs per launch.

Tolerance, elementwise: |error| <= n_r 2^-23 (|A| |B|)[r, n] (exact products in
FP32 sums of any order), 2^-23 |result| for beta, plus 2^-11 |ref| + 2^-24 for
FP16 output; E4M3 against its dequantized operands with 2^-21 |ref| for the two
scale products."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import tca_spmm  # noqa: E402


def matrix(M, K, long_row, N, seed):
    rng = np.random.default_rng(seed)
    n = np.full(M, K // 4)
    n[M // 128 * 128:] = long_row  # the last window
    n[-1] = 0
    rp = np.concatenate([[0], np.cumsum(n)]).astype(np.int32)
    col = np.concatenate([np.sort(rng.choice(K, k, replace=False)) for k in n]).astype(np.int32)
    return dict(M=M, K=K, N=N, row_ptr=rp, col=col, vals=rng.standard_normal(col.size).astype(np.float16),
                B=rng.uniform(-1, 1, (K, N)).astype(np.float16))


CASES = [(130, 2000, 33), (131, 3000, 200), (257, 700, 100), (5, 900, 640), (1, 4000, 4000)]


@pytest.mark.parametrize("M,K,long_row", CASES)
@pytest.mark.parametrize("N", [32, 128, 264, 624])
@pytest.mark.parametrize("out", ["f16", "f32"])
def test_long_rows(cuda, M, K, long_row, N, out):
    c = matrix(M, K, min(long_row, K), N, M + K + N)
    rp, ci, v, B = (torch.from_numpy(c[k]).to(cuda) for k in ("row_ptr", "col", "vals", "B"))
    dt = torch.float16 if out == "f16" else torch.float32
    n_r = np.diff(c["row_ptr"])[:, None]
    ref = oracle.spmm_f64(c["row_ptr"], c["col"], c["vals"], c["B"])
    mag = oracle.spmm_f64(c["row_ptr"], c["col"], np.abs(c["vals"]), np.abs(c["B"]))
    half = (lambda x: 2.0 ** -11 * np.abs(x) + 2.0 ** -24) if out == "f16" else (lambda x: 0)
    for path in ("auto", "cuda_core"):
        plan = tca_spmm.Plan(rp, ci, v, K, path=path)
        C = torch.full((M, N), 3.0, dtype=dt, device=cuda)
        plan.spmm(B, out=C)
        assert np.all(np.abs(C.cpu().numpy().astype(np.float64) - ref) <= n_r * 2.0 ** -23 * mag + half(ref))
        want = np.where(n_r > 0, 2 * ref + 0.25, 0.5)
        tol = 2 * n_r * 2.0 ** -23 * mag + 2.0 ** -23 * np.abs(want) + half(want)
        outs = [torch.full((M, N), 0.5, dtype=dt, device=cuda) for _ in range(3)]
        tca_spmm.spmm_batched([plan] * 3, [B] * 3, outs, alpha=2.0, beta=0.5, keep_empty_rows=True)
        for C in outs:
            assert np.all(np.abs(C.cpu().numpy().astype(np.float64) - want) <= tol)
        C = torch.full((M, N), 3.0, dtype=dt, device=cuda)
        tca_spmm.spmm_batched([plan], [B], [C], cc_cols=2)
        assert np.all(np.abs(C.cpu().numpy().astype(np.float64) - ref) <= n_r * 2.0 ** -23 * mag + half(ref))
        plan.status()


@pytest.mark.parametrize("M,K,long_row", CASES)
@pytest.mark.parametrize("N", [32, 264, 624])
def test_long_rows_e4m3(cuda, M, K, long_row, N):
    c = matrix(M, K, min(long_row, K), N, M + K + N)
    rp, ci, v, B = (torch.from_numpy(c[k]).to(cuda) for k in ("row_ptr", "col", "vals", "B"))
    n_r = np.diff(c["row_ptr"])[:, None]
    ref = oracle.spmm_fp8_f64(c["row_ptr"], c["col"], c["vals"], c["B"])
    mag = oracle.spmm_f64(c["row_ptr"], c["col"], np.abs(c["vals"]) * np.float16(1.0625),
                          np.abs(c["B"]) * np.float16(1.0625))
    C = tca_spmm.Plan(rp, ci, v, K).spmm_fp8(B, out_dtype=torch.float32)
    assert np.all(np.abs(C.cpu().numpy().astype(np.float64) - ref) <= n_r * 2.0 ** -23 * mag + 2.0 ** -21 * np.abs(ref))
