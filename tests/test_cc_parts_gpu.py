"""CUDA-core items whose rows are cut among warps: halves where there are a few
rounds of items (2,368 to 9,472) and N takes several passes, or an item has many
rows; up to four parts where there are fewer; items of one row among them, rows
without nonzeros, alpha and beta, a batch of plans with different row lengths.

Tolerance, elementwise: |error| <= n_r 2^-23 (|A| |B|)[r, n] (exact products in
FP32 sums of any order), twice that with alpha = 2, and 2^-23 |result| for
beta; E4M3 against its dequantized operands with 2^-21 |ref| for the two scale
products."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import tca_spmm  # noqa: E402


def matrix(M, lengths, K, N, seed):
    rng = np.random.default_rng(seed)
    n = np.resize(np.array(lengths), M)
    rp = np.concatenate([[0], np.cumsum(n)]).astype(np.int32)
    col = np.concatenate([np.sort(rng.choice(K, k, replace=False)) for k in n]).astype(np.int32)
    return dict(M=M, K=K, N=N, row_ptr=rp, col=col, vals=(rng.standard_normal(col.size) * 0.1).astype(np.float16),
                B=rng.uniform(-1, 1, (K, N)).astype(np.float16))


CASES = [(2500, [24], 264), (5000, [16], 520), (3000, [40, 3, 0, 9], 1032), (40000, [2, 2, 1], 136), (700, [5, 30], 72),
         (75000, [1], 256)]


@pytest.mark.parametrize("M,lengths,N", CASES)
@pytest.mark.parametrize("sort_rows", [False, True])
def test_parts(cuda, M, lengths, N, sort_rows):
    c = matrix(M, lengths, 300, N, M + N)
    rp, ci, v, B = (torch.from_numpy(c[k]).to(cuda) for k in ("row_ptr", "col", "vals", "B"))
    n_r = np.diff(c["row_ptr"])[:, None]
    ref = oracle.spmm_f64(c["row_ptr"], c["col"], c["vals"], c["B"])
    mag = oracle.spmm_f64(c["row_ptr"], c["col"], np.abs(c["vals"]), np.abs(c["B"]))
    plan = tca_spmm.Plan(rp, ci, v, c["K"], path="cuda_core", sort_rows=sort_rows)
    want = np.where(n_r > 0, 2 * ref + 0.25, 0.5)
    C = torch.full((M, N), 0.5, device=cuda)
    plan.spmm(B, out=C, alpha=2.0, beta=0.5, keep_empty_rows=True)
    assert np.all(np.abs(C.cpu().numpy().astype(np.float64) - want) <= 2 * n_r * 2.0 ** -23 * mag + 2.0 ** -23 * np.abs(want))
    small = matrix(300, [12, 0, 31], 300, N, 1)
    d = [torch.from_numpy(small[k]).to(cuda) for k in ("row_ptr", "col", "vals", "B")]
    p2 = tca_spmm.Plan(*d[:3], 300, path="cuda_core")
    outs = [torch.full((M, N), 3.0, device=cuda), torch.full((300, N), 3.0, device=cuda)]
    tca_spmm.spmm_batched([plan, p2], [B, d[3]], outs)
    assert np.all(np.abs(outs[0].cpu().numpy() - ref) <= n_r * 2.0 ** -23 * mag)
    ref2 = oracle.spmm_f64(small["row_ptr"], small["col"], small["vals"], small["B"])
    mag2 = oracle.spmm_f64(small["row_ptr"], small["col"], np.abs(small["vals"]), np.abs(small["B"]))
    assert np.all(np.abs(outs[1].cpu().numpy() - ref2) <= np.diff(small["row_ptr"])[:, None] * 2.0 ** -23 * mag2)
    C = plan.spmm_fp8(B, out_dtype=torch.float32)
    ref8 = oracle.spmm_fp8_f64(c["row_ptr"], c["col"], c["vals"], c["B"])
    mag8 = mag * 1.0625 ** 2  # the quantized operands' magnitudes exceed the FP16 ones by at most 2^-4 each
    assert np.all(np.abs(C.cpu().numpy() - ref8) <= n_r * 2.0 ** -23 * mag8 + 2.0 ** -21 * np.abs(ref8))
