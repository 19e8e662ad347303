"""Plan-free forwards of as many rows as a 32-bit count holds: row numbers and
the search over the rows must not pass the largest int on the way."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import tca_spmm  # noqa: E402


@pytest.mark.parametrize("N", [8, 1])  # the short rows kernel; the rows kernel (two-byte accesses)
def test_rows_near_the_largest_int(cuda, N):
    if torch.cuda.mem_get_info()[0] < 64 << 30:
        pytest.skip("needs 64 GB of device memory")
    M = 2 ** 31 - 2
    row_ptr = torch.zeros(M + 1, dtype=torch.int32, device=cuda)  # one nonzero in the first row, one in the last
    row_ptr[1:] = 1
    row_ptr[M] = 2
    col = torch.tensor([1, 2], dtype=torch.int32, device=cuda)
    vals = torch.tensor([2.0, 3.0], dtype=torch.float16, device=cuda)
    B = torch.arange(1, 3 * N + 1, device=cuda).reshape(3, N).half()
    C = torch.full((M, N), 7.0, dtype=torch.float16, device=cuda)
    tca_spmm.spmm_csr(row_ptr, col, vals, B, K=3, out=C)
    assert torch.equal(C[0], 2 * B[1]) and torch.equal(C[M - 1], 3 * B[2])
    for lo in range(1, M - 1, 1 << 28):
        assert not C[lo:min(M - 1, lo + (1 << 28))].any()
    del row_ptr, C
    torch.cuda.empty_cache()
