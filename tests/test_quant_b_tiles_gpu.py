"""B's E4M3 quantization over tiles (large matrices), around the sizes where it
takes over from the clusters: ragged tiles, rows of B that are not 16-byte
aligned, all-zero columns, and a batch of large and small matrices -- bytes and
scales equal to the oracle's bit for bit (of the batch: the same results as one
by one)."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import tca_spmm  # noqa: E402


def matrix(K, N, seed):
    rng = np.random.default_rng(seed)
    B = (rng.standard_normal((K, N), dtype=np.float32) * np.exp(rng.uniform(-6, 6, N)).astype(np.float32))
    B = B.clip(-6e4, 6e4).astype(np.float16)
    B[:, N // 2] = 0
    return B


@pytest.mark.parametrize("K,N", [(6145, 1024), (8191, 1016), (20001, 257), (41000, 136), (90000, 24), (4096, 4096), (1025, 17000)])
@pytest.mark.parametrize("pad", [0, 1])
def test_quant_b_tiles(cuda, K, N, pad):
    Bh = matrix(K, N, K + N)
    wide = torch.zeros((K, N + pad), dtype=torch.float16, device=cuda)
    wide[:, :N] = torch.from_numpy(Bh).to(cuda)
    want_q, want_s = oracle.quant_cols(Bh)
    for _ in range(2):  # the maxima are cleared in every call
        q, s = tca_spmm.quantize_b_fp8(wide[:, :N])
        assert np.array_equal(s.cpu().numpy(), want_s[:N])
        assert np.array_equal(q.cpu().numpy()[:, :N], np.asarray(want_q)[:, :N])


def test_batch_of_large_and_small(cuda):
    rng = np.random.default_rng(3)
    plans, Bs, outs, single = [], [], [], []
    for K, N in ((9000, 1024), (70, 64), (3000, 1016), (9000, 8), (1, 256)):
        M = 40
        rows = [np.sort(rng.choice(K, min(K, 30), replace=False)) for _ in range(M)]
        rp = np.concatenate([[0], np.cumsum([r.size for r in rows])]).astype(np.int32)
        col = np.concatenate(rows).astype(np.int32)
        v = rng.standard_normal(col.size).astype(np.float16)
        p = tca_spmm.Plan(*(torch.from_numpy(x).to(cuda) for x in (rp, col, v)), K)
        p.quantize_fp8()
        plans.append(p)
        Bs.append(torch.from_numpy(matrix(K, N, K)).to(cuda))
        outs.append(torch.empty((M, N), device=cuda))
        single.append(p.spmm_fp8(Bs[-1], out_dtype=torch.float32))
    tca_spmm.spmm_fp8_batched(plans, Bs, outs)
    for a, b in zip(outs, single):
        assert torch.allclose(a, b, rtol=2.0 ** -18, atol=2.0 ** -18 * b.abs().max().item())
