"""The rows kernel on row offsets that are not increasing: every row is clamped
to [0, nnz] by itself and written once, whatever the others are. The sums are
small whole numbers, exact in FP32 in any order: results are compared exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import tca_spmm  # noqa: E402


def expected(row_ptr, col, vals, B):
    """Row sums from prefix sums over the nonzeros."""
    nnz = col.size
    pre = np.zeros((nnz + 1, B.shape[1]))
    for n in range(B.shape[1]):
        np.cumsum(vals.astype(np.float64) * B[col, n], out=pre[1:, n])
    start = np.clip(row_ptr[:-1].astype(np.int64), 0, nnz)
    end = np.maximum(start, np.clip(row_ptr[1:].astype(np.int64), 0, nnz))
    return pre[end] - pre[start], end > start


@pytest.mark.parametrize("M,N", [(700, 24), (5000, 136), (3000, 23)])
@pytest.mark.parametrize("order", ["random", "alternating", "decreasing", "some wrong"])
def test_each_row_once(cuda, M, N, order):
    rng = np.random.default_rng(M + N)
    nnz, K = 40 * M, 60  # more than 32 a row as the call counts them: the rows kernel
    if order == "random":
        row_ptr = rng.integers(-30, 150, M + 1) + np.repeat(rng.integers(0, nnz, M // 50 + 1), 50)[:M + 1]
        if row_ptr.size < M + 1:
            row_ptr = np.concatenate([row_ptr, np.zeros(M + 1 - row_ptr.size, np.int64)])
    elif order == "alternating":
        row_ptr = np.arange(M + 1) % 2 * 300
    elif order == "decreasing":
        row_ptr = np.arange(M + 1)[::-1] * 40
    else:
        row_ptr = np.arange(M + 1) * 40
        row_ptr[rng.choice(M + 1, M // 20, replace=False)] += rng.integers(-500, 500, M // 20)
    row_ptr = row_ptr.astype(np.int32)
    col = rng.integers(0, K, nnz).astype(np.int32)
    vals = rng.integers(-2, 3, nnz).astype(np.float16)
    B = rng.integers(-2, 3, (K, N)).astype(np.float16)
    ref, some = expected(row_ptr, col, vals, B.astype(np.float64))
    dev = [torch.from_numpy(x).to(cuda) for x in (row_ptr, col, vals, B)]
    C = torch.full((M, N), 4.0, dtype=torch.float32, device=cuda)
    tca_spmm.spmm_csr(*dev, K=K, out=C, alpha=1.0, beta=0.5, keep_empty_rows=True)
    want = np.where(some[:, None], ref + 2.0, 4.0)
    assert np.array_equal(C.cpu().numpy().astype(np.float64), want)


def test_overlapping_rows_beyond_32_bits(cuda):
    """520 overlapping rows of 8.4 million nonzeros: a block's rows hold more
    nonzeros together than a 32-bit sum."""
    rng = np.random.default_rng(1)
    M, K, N, nnz = 520, 64, 8, 8_400_000
    row_ptr = (np.arange(M + 1) % 2 * nnz).astype(np.int32)
    col = rng.integers(0, K, nnz).astype(np.int32)
    vals = (rng.random(nnz) < 2.0 ** -10).astype(np.float16)
    B = rng.integers(-2, 3, (K, N)).astype(np.float16)
    ref, _ = expected(row_ptr, col, vals, B.astype(np.float64))
    dev = [torch.from_numpy(x).to(cuda) for x in (row_ptr, col, vals, B)]
    around = torch.full((M + 1040, N), 3.0, dtype=torch.float32, device=cuda)  # rows before and after C
    C = around[520:520 + M]
    tca_spmm.spmm_csr(*dev, K=K, out=C)
    got = around.cpu().numpy()
    assert np.all(got[:520] == 3.0) and np.all(got[520 + M:] == 3.0)
    assert np.array_equal(got[520:520 + M].astype(np.float64), ref)
