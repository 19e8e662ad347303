"""B's E4M3 quantization in one launch: clusters of 1 to 8 blocks, strips of 64,
16 and 8 columns, rows that fit shared memory and not, ragged K and N, rows of
B that are not 16-byte aligned, all-zero columns -- bytes and scales equal to
the oracle's bit for bit."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import tca_spmm  # noqa: E402


@pytest.mark.parametrize("K,N", [(1, 8), (63, 64), (130, 72), (257, 200), (1024, 256), (4096, 72), (4100, 136),
                                 (9000, 24), (20000, 40), (110000, 8)])
@pytest.mark.parametrize("pad", [0, 1])
def test_quant_b(cuda, K, N, pad):
    rng = np.random.default_rng(K + N)
    Bh = (rng.standard_normal((K, N)) * np.exp(rng.uniform(-6, 6, N))).clip(-6e4, 6e4).astype(np.float16)
    Bh[:, N // 2] = 0
    wide = torch.zeros((K, N + pad), dtype=torch.float16, device=cuda)
    wide[:, :N] = torch.from_numpy(Bh).to(cuda)
    q, s = tca_spmm.quantize_b_fp8(wide[:, :N])
    want_q, want_s = oracle.quant_cols(Bh)
    assert np.array_equal(s.cpu().numpy(), want_s[:N])
    assert np.array_equal(q.cpu().numpy()[:, :N], np.asarray(want_q)[:, :N])
