"""The rows kernel (plan-free forward, and planned forwards whose operands are
not 16-byte aligned): rows cut into equal runs over the groups of a block.
Edges: one row, a row longer than a block's whole run, runs inside one row,
leading / trailing / only empty rows, more rows than fit shared memory at a
time, every column width of a group, N of one column.

Tolerance, elementwise: exact products accumulated in FP32 in any order,
|error| <= n_r 2^-23 (|A| |B|)[r, n], plus 2^-11 |ref| + 2^-24 for FP16 output."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import tca_spmm  # noqa: E402


def rows_case(kind, rng):
    if kind == "one_row":
        return np.array([700])
    if kind == "one_full":  # one long row among short ones
        n = rng.integers(0, 3, 500)
        n[137] = 900
        return n
    if kind == "sorted":  # long rows first
        return np.sort(rng.zipf(1.4, 600).clip(0, 900))[::-1]
    if kind == "empty_ends":
        n = rng.integers(0, 40, 300)
        n[:100] = 0
        n[-90:] = 0
        return n
    if kind == "all_empty":
        return np.zeros(70, int)
    if kind == "many_short":  # more rows per block than shared memory holds
        return rng.integers(0, 2, 40000)
    return rng.integers(20, 60, 257)


def make(kind, N, seed):
    rng = np.random.default_rng(seed)
    K = 901
    n = np.asarray(rows_case(kind, rng), dtype=np.int64)
    row_ptr = np.concatenate([[0], np.cumsum(n)]).astype(np.int32)
    col = np.concatenate([np.sort(rng.choice(K, k, replace=False)) for k in n] + [np.zeros(0, int)]).astype(np.int32)
    vals = rng.standard_normal(col.size).astype(np.float16)
    return dict(M=n.size, K=K, N=N, row_ptr=row_ptr, col=col, vals=vals,
                B=rng.uniform(-1, 1, (K, N)).astype(np.float16))


KINDS = ["one_row", "one_full", "sorted", "empty_ends", "all_empty", "many_short", "even"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("N", [1, 8, 33, 40, 100, 136, 203, 264])
@pytest.mark.parametrize("out", ["f16", "f32"])
def test_rows(cuda, kind, N, out):
    c = make(kind, N, 7 * N + len(kind))
    rp, ci, v, B = (torch.from_numpy(c[k]).to(cuda) for k in ("row_ptr", "col", "vals", "B"))
    dt = torch.float16 if out == "f16" else torch.float32
    ref = oracle.spmm_f64(c["row_ptr"], c["col"], c["vals"], c["B"])
    mag = oracle.spmm_f64(c["row_ptr"], c["col"], np.abs(c["vals"]), np.abs(c["B"]))
    n_r = np.diff(c["row_ptr"])[:, None]
    tol = n_r * 2.0 ** -23 * mag + (2.0 ** -11 * np.abs(ref) + 2.0 ** -24 if out == "f16" else 0)
    runs = [lambda o, **kw: tca_spmm.spmm_csr(rp, ci, v, B, out=o, **kw)]
    if N % 8:
        plan = tca_spmm.Plan(rp, ci, v, c["K"])
        runs.append(lambda o, **kw: plan.spmm(B, out=o, **kw))
    for run in runs:
        C = torch.full((c["M"], N), 3.0, dtype=dt, device=cuda)
        run(C)
        assert np.all(np.abs(C.cpu().numpy().astype(np.float64) - ref) <= tol)
        # beta != 0, rows without nonzeros untouched: alpha, beta exact powers of two
        C = torch.full((c["M"], N), 0.5, dtype=dt, device=cuda)
        run(C, alpha=2.0, beta=0.5, keep_empty_rows=True)
        want = np.where(n_r > 0, 2 * ref + 0.25, 0.5)
        extra = 2.0 ** -23 * np.abs(want) + (2.0 ** -11 * np.abs(want) + 2.0 ** -24 if out == "f16" else 0)
        assert np.all(np.abs(C.cpu().numpy().astype(np.float64) - want) <= 2 * n_r * 2.0 ** -23 * mag + extra)


def test_rows_malformed(cuda):
    """Row offsets and columns out of range: rows are clamped one by one, such
    nonzeros add nothing, also over infinite rows of B."""
    rp = torch.tensor([0, 5, 3, 90, 40, 12], dtype=torch.int32, device=cuda)
    ci = torch.tensor([0, 1, -4, 7, 99, 2, 3, 1, 0, 2], dtype=torch.int32, device=cuda)
    v = torch.ones(10, dtype=torch.float16, device=cuda)
    B = torch.ones((8, 24), dtype=torch.float16, device=cuda)
    B[0] = float("inf")
    for N in (24, 23):
        C = tca_spmm.spmm_csr(rp, ci, v, B[:, :N].contiguous(), K=8, out_dtype=torch.float32)
        torch.cuda.synchronize()
        assert C.shape == (5, N)


@pytest.mark.parametrize("N", [64, 128, 136, 256])
@pytest.mark.parametrize("per_row", [20, 100])  # the short rows kernel, the rows kernel
def test_rows_malformed_columns(cuda, N, per_row):
    """Columns out of range among valid ones, at the start, inside and at the end
    of a row: they add nothing, also over infinite rows of B; the others add up."""
    rng = np.random.default_rng(N + per_row)
    M, K = 37, 300
    col = np.concatenate([np.sort(rng.choice(np.arange(1, K), per_row, replace=False)) for _ in range(M)])
    col = col.astype(np.int32)
    bad = rng.random(col.size) < 0.04
    bad[[0, per_row, col.size - 1]] = True
    bad[5 * per_row:9 * per_row] = False
    ok = np.where(bad, 0, col)
    col[bad] = rng.choice([-1, K, -2 ** 31, 2 ** 31 - 1], bad.sum())
    vals = rng.standard_normal(col.size).astype(np.float16)
    B = rng.uniform(-1, 1, (K, N)).astype(np.float16)
    A = np.zeros((M, K))
    A[np.repeat(np.arange(M), per_row)[~bad], ok[~bad]] = vals[~bad]
    ref, mag = A @ B.astype(np.float64), np.abs(A) @ np.abs(B.astype(np.float64))
    B[0] = np.inf  # no valid nonzero has column 0
    rp = torch.arange(0, M * per_row + 1, per_row, dtype=torch.int32, device=cuda)
    dev = [torch.from_numpy(x).to(cuda) for x in (col, vals, B)]
    C = tca_spmm.spmm_csr(rp, *dev, K=K, out_dtype=torch.float32)
    assert np.all(np.abs(C.cpu().numpy() - ref) <= per_row * 2.0 ** -23 * mag)
