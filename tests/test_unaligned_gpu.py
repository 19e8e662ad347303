"""Forwards whose operands do not allow 16-byte accesses: through a padded copy
of B (nnz * N from 2^25 on), on the tensor cores (a plan, FP16 C) or the rows
kernel (FP32 C, plan-free), and below that size, and under stream capture,
straight. Odd N, N of whole slabs with unaligned B, aligned B with unaligned C,
more than one 256-column slice, rows without nonzeros, alpha and beta.

Tolerance, elementwise: as for the aligned kernels, |error| <= n_r 2^-23
(|A| |B|)[r, n] (FP32 accumulation of exact products), one FP32 rounding more
for beta (2^-23 of the result), plus 2^-11 |ref| + 2^-24 for FP16 output."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import tca_spmm  # noqa: E402


def case(M, K, N, density, cuda, seed):
    rng = np.random.default_rng(seed)
    mask = rng.random((M, K)) < density
    mask[rng.random(M) < 0.1] = False
    rows, cols = np.nonzero(mask)
    rp = np.concatenate([[0], np.cumsum(mask.sum(1))]).astype(np.int32)
    vals = rng.standard_normal(cols.size).astype(np.float16)
    B = rng.uniform(-1, 1, (K, N)).astype(np.float16)
    A = np.zeros((M, K))
    A[rows, cols] = vals
    dev = [torch.from_numpy(x).to(cuda) for x in (rp, cols.astype(np.int32), vals)]
    return dev, B, A, mask.sum(1)[:, None]


SHAPES = [(700, 1100, 99, 0.5), (513, 770, 264, 0.4), (900, 400, 513, 0.3), (1300, 900, 35, 0.9), (300, 300, 129, 0.3)]


@pytest.mark.parametrize("M,K,N,density", SHAPES)
@pytest.mark.parametrize("out", ["f16", "f32"])
@pytest.mark.parametrize("place", ["as_is", "b_off", "c_off"])
def test_unaligned(cuda, M, K, N, density, out, place):
    (rp, ci, v), Bh, A, n_r = case(M, K, N, density, cuda, M + N)
    # 1300 x 900 lies just below the size from which B is copied, 300 x 300 far below
    assert (ci.numel() * N >= 2 ** 25) == ((M, K) not in ((300, 300), (1300, 900)))
    dt = torch.float16 if out == "f16" else torch.float32
    B = torch.from_numpy(Bh).to(cuda)
    if place == "b_off":  # rows of B at odd offsets
        wide = torch.zeros((K, N + 3), dtype=torch.float16, device=cuda)
        wide[:, 1:N + 1] = B
        B = wide[:, 1:N + 1]

    def target(value):
        if place == "c_off":
            t = torch.full((M, N + 3), value, dtype=dt, device=cuda)
            return t, t[:, 1:N + 1]
        t = torch.full((M, N), value, dtype=dt, device=cuda)
        return t, t

    b64 = Bh.astype(np.float64)
    ref, mag = A @ b64, np.abs(A) @ np.abs(b64)
    half = (lambda x: 2.0 ** -11 * np.abs(x) + 2.0 ** -24) if out == "f16" else (lambda x: 0)
    plan = tca_spmm.Plan(rp, ci, v, K)
    for f in (plan.spmm, lambda B, **kw: tca_spmm.spmm_csr(rp, ci, v, B, **kw)):
        whole, C = target(3.0)
        f(B, out=C)
        assert np.all(np.abs(C.cpu().numpy().astype(np.float64) - ref) <= n_r * 2.0 ** -23 * mag + half(ref))
        if place == "c_off":  # nothing outside C is written
            assert (whole[:, 0] == 3).all() and (whole[:, N + 1:] == 3).all()
        whole, C = target(0.5)
        f(B, out=C, alpha=2.0, beta=0.5, keep_empty_rows=True)
        want = np.where(n_r > 0, 2 * ref + 0.25, 0.5)
        tol = 2 * n_r * 2.0 ** -23 * mag + 2.0 ** -23 * np.abs(want) + half(want)
        assert np.all(np.abs(C.cpu().numpy().astype(np.float64) - want) <= tol)
    plan.status()


def test_unaligned_capture(cuda):
    (rp, ci, v), Bh, A, n_r = case(700, 1100, 99, 0.5, cuda, 3)
    plan = tca_spmm.Plan(rp, ci, v, 1100)
    B = torch.from_numpy(Bh).to(cuda)
    C = torch.empty((700, 99), dtype=torch.float16, device=cuda)
    used = tca_spmm.pool_stats()["used"]
    plan.spmm(B, out=C)  # with the copy
    torch.cuda.synchronize()
    assert tca_spmm.pool_stats()["used"] == used  # given back
    eager = C.clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        plan.spmm(B, out=C)
    C.zero_()
    g.replay()
    torch.cuda.synchronize()
    mag = np.abs(A) @ np.abs(Bh.astype(np.float64))
    d = np.abs(C.cpu().numpy().astype(np.float64) - eager.cpu().numpy())
    assert np.all(d <= 2 * n_r * 2.0 ** -23 * mag + 2.0 ** -10 * np.abs(A @ Bh.astype(np.float64)) + 2.0 ** -23)


@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("out", ["f16", "f32"])
def test_unaligned_nonfinite(cuda, bad, out):
    """An infinity or NaN in B reaches the rows that hold a nonzero of its
    column and no other, as in forwards without a copy."""
    M, K, N = 700, 1100, 99
    (rp, ci, v), Bh, A, n_r = case(M, K, N, 0.5, cuda, 5)
    clean = np.zeros((M, N), dtype=bool)
    clean[:] = (A[:, 17] == 0)[:, None]
    clean[:, np.arange(N) != 40] = True
    b64 = Bh.astype(np.float64)
    ref, mag = A @ b64, np.abs(A) @ np.abs(b64)
    Bh[17, 40] = bad
    dt = torch.float16 if out == "f16" else torch.float32
    C = torch.full((M, N), 0.5, dtype=dt, device=cuda)
    tca_spmm.Plan(rp, ci, v, K).spmm(torch.from_numpy(Bh).to(cuda), out=C, alpha=2.0, beta=0.5)
    got, want = C.cpu().numpy().astype(np.float64), 2 * ref + 0.25
    tol = 2 * n_r * 2.0 ** -23 * mag + 2.0 ** -23 * np.abs(want)
    if out == "f16":
        tol = tol + 2.0 ** -11 * np.abs(want) + 2.0 ** -24
    assert np.all(np.abs(got - want)[clean] <= tol[clean])
    hit = got[~clean]
    assert hit.size and not np.isfinite(hit).any()
    if np.isinf(bad):
        assert np.all(np.sign(hit) == np.sign(bad * A[:, 17][A[:, 17] != 0]))
