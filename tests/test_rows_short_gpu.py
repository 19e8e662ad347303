"""The plan-free short rows kernel where a block holds none, one, several or
only long rows (more than 64 nonzeros): its groups are dealt to them by length.

Tolerance, elementwise: |error| <= n_r 2^-23 (|A| |B|)[r, n], twice that with
alpha = 2, 2^-23 |result| for beta (exact products in FP32 sums of any order)."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import tca_spmm  # noqa: E402

LENGTHS = {
    "one": lambda rng, M: np.where(np.arange(M) == M // 2, 3000, 2),
    "some": lambda rng, M: np.where(rng.random(M) < 0.04, rng.integers(65, 400, M), 3),
    "unequal": lambda rng, M: np.where(rng.random(M) < 0.06, np.where(rng.random(M) < 0.2, 2500, 66), rng.integers(0, 3, M)),
    "first block only": lambda rng, M: np.where(np.arange(M) % ((M + 15) // 16) == 0, 100, 1),
}


@pytest.mark.parametrize("law", sorted(LENGTHS))
@pytest.mark.parametrize("M", [1, 40, 1500])
@pytest.mark.parametrize("N", [8, 32, 64, 96, 256, 272])
def test_long_rows_among_short_ones(cuda, law, M, N):
    rng = np.random.default_rng(M + N)
    K = 3000
    n = LENGTHS[law](rng, M)
    if n.sum() > 32 * M:  # keep the mean that selects this kernel: rows without nonzeros after them
        n = np.concatenate([n, np.zeros(int(n.sum() // 32) + 1 - M, n.dtype)])
    row_ptr = np.concatenate([[0], np.cumsum(n)]).astype(np.int32)
    col = np.concatenate([np.sort(rng.choice(K, k, replace=False)) for k in n]).astype(np.int32)
    vals = rng.standard_normal(col.size).astype(np.float16)
    B = rng.uniform(-1, 1, (K, N)).astype(np.float16)
    ref = oracle.spmm_f64(row_ptr, col, vals, B)
    mag = oracle.spmm_f64(row_ptr, col, np.abs(vals), np.abs(B))
    dev = [torch.from_numpy(x).to(cuda) for x in (row_ptr, col, vals, B)]
    n_r = n[:, None]
    C = torch.full((n.size, N), 3.0, device=cuda)
    tca_spmm.spmm_csr(*dev, K=K, out=C)
    assert np.all(np.abs(C.cpu().numpy() - ref) <= n_r * 2.0 ** -23 * mag)
    again = torch.empty_like(C)
    tca_spmm.spmm_csr(*dev, K=K, out=again)
    assert torch.equal(C, again)
    want = np.where(n_r > 0, 2 * ref + 0.25, 0.5)
    C = torch.full((n.size, N), 0.5, device=cuda)
    tca_spmm.spmm_csr(*dev, K=K, out=C, alpha=2.0, beta=0.5, keep_empty_rows=True)
    assert np.all(np.abs(C.cpu().numpy() - want) <= 2 * n_r * 2.0 ** -23 * mag + 2.0 ** -23 * np.abs(want))
