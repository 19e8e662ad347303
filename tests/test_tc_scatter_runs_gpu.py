"""Runs of condensed sparse chunks, whose rows of B the scatter warps gather,
before and between chunks that the loader of B issues itself (64 consecutive
columns, or a condensed chunk with a tile image): runs longer than the ring's
stages (at most 11) several times over, at the start of a CTA's chunks and
after others, within a window (whose walk starts at another chunk per window)
and from one item of a CTA to the next.

Tolerance, elementwise, as in test_tc_ring_gpu.py: n_r 2^-23 (|A| |B|)[r, n]
for a row of n_r nonzeros summed in FP32 in any order, plus 2^-11 |ref| +
2^-24 for FP16 output, and with E4M3 2^-21 |ref| for the two scale products."""
import numpy as np
import pytest

from oracle import oracle
from tca_spmm import gen

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import tca_spmm  # noqa: E402


def csr(mask_rows, K, rng, N):
    """Rows given as sorted column arrays."""
    row_ptr = np.concatenate([[0], np.cumsum([len(r) for r in mask_rows])]).astype(np.int32)
    col = np.concatenate(mask_rows).astype(np.int32)
    vals = (rng.standard_normal(col.size) * 0.1).astype(np.float16)
    return dict(M=len(mask_rows), K=K, N=N, row_ptr=row_ptr, col=col, vals=vals, B=gen.uniform_b(rng, K, N))


def window_rows(rng, chunks):
    """128 rows over condensed chunks of 64 distinct columns each, ascending,
    one letter per chunk: 's' two nonzeros per column, spread columns (a sparse
    chunk); 'i' 24 rows use each column (an image); 'd' 64 consecutive columns,
    two nonzeros each. Returns the rows and K."""
    rows = [[] for _ in range(128)]
    base = 0
    for kind in chunks:
        if kind == "d":
            cols = base + np.arange(64)
            base += 64
        else:
            cols = base + np.sort(rng.choice(320, 64, replace=False))
            base += 320
        for c in cols:
            for r in rng.choice(128, 24 if kind == "i" else 2, replace=False):
                rows[r].append(int(c))
    return [np.array(r, np.int32) for r in rows], base


def check(got, ref, c, f16, f8=False):
    n_r = np.diff(c["row_ptr"])[:, None]
    up = np.float16(1.0625) if f8 else np.float16(1)  # E4M3 operands exceed the FP16 ones by at most 2^-4 each
    mag = oracle.spmm_f64(c["row_ptr"], c["col"], np.abs(c["vals"]) * up, np.abs(c["B"]) * up)
    tol = n_r * 2.0 ** -23 * mag + (2.0 ** -21 * np.abs(ref) if f8 else 0.0)
    if f16:
        tol = tol + 2.0 ** -11 * np.abs(ref) + 2.0 ** -24
    assert np.all(np.abs(got.cpu().numpy().astype(np.float64) - ref) <= tol)


def on_gpu(c, cuda, **opts):
    rp, ci, v, B = (torch.from_numpy(c[k]).to(cuda) for k in ("row_ptr", "col", "vals", "B"))
    return tca_spmm.Plan(rp, ci, v, c["K"], **opts), B


def chunk_kinds(c):
    """The letters of the chunks that the plan has, per tensor-core window."""
    p = oracle.build_plan(c["row_ptr"], c["col"], c["vals"], c["K"], sort_rows=False, path=2)
    out = []
    for t in range(p["n_tc"]):
        k = ""
        for ch in range(p["tile_first"][t], p["tile_first"][t + 1]):
            cols = p["win_cols"][ch * 64:(ch + 1) * 64]
            direct = cols[0] >= 0 and cols[63] == cols[0] + 63
            k += "d" if direct else "i" if p["tile_ptr"][ch + 1] - p["tile_ptr"][ch] >= 512 else "s"
        out.append(k)
    return out


WALKS = ["s" * 33 + "d", "s" * 33 + "i", "s" * 8 + "d" + "s" * 13 + "i" + "s" * 23 + "d" * 5, "i" + "s" * 40 + "d" * 12]


@pytest.mark.parametrize("walk", range(len(WALKS)))
@pytest.mark.parametrize("N,n_tile", [(64, 64), (128, 128), (256, 256), (200, 256)])
@pytest.mark.parametrize("precision", ["f16", "e4m3"])
def test_runs_in_a_window(cuda, walk, N, n_tile, precision):
    rng = np.random.default_rng(100 + walk)
    rows, K = window_rows(rng, WALKS[walk])
    for _ in range(2):  # two more windows of the same columns, whose walks start one and two chunks later
        rows = rows + [rows[r] for r in rng.permutation(128)]
    c = csr(rows, K, rng, N)
    assert chunk_kinds(c) == [WALKS[walk]] * 3
    plan, B = on_gpu(c, cuda, path="tensor_core", sort_rows=False)
    C = torch.full((c["M"], N), 7.0, dtype=torch.float16, device=cuda)
    if precision == "e4m3":
        tca_spmm.spmm_fp8_batched([plan], [B], [C], n_tile=max(n_tile, 128))
        ref = oracle.spmm_fp8_f64(c["row_ptr"], c["col"], c["vals"], c["B"])
    else:
        tca_spmm.spmm_batched([plan], [B], [C], n_tile=n_tile)
        ref = oracle.spmm_f64(c["row_ptr"], c["col"], c["vals"], c["B"])
    plan.status()
    check(C, ref, c, True, precision == "e4m3")


@pytest.mark.parametrize("later", ["d" * 34, "d" * 3])  # as many chunks per item (round-robin), or fewer (dealt out)
@pytest.mark.parametrize("precision", ["f16", "e4m3"])
def test_runs_between_items(cuda, later, precision):
    """More items than CTAs: items of condensed sparse chunks, then items of
    64-column blocks of K on the same CTAs."""
    rng = np.random.default_rng(len(later))
    N, n_tile = (1024, 64) if precision == "f16" else (1024, 128)
    windows = 10 if precision == "f16" else 20
    cs = []
    for walk in ("s" * 34, later):
        rows, K = window_rows(rng, walk)
        rows = [rows[r] for _ in range(windows) for r in rng.permutation(128)]
        cs.append(csr(rows, K, rng, N))
    assert set(chunk_kinds(cs[0])) == {"s" * 34} and set(chunk_kinds(cs[1])) == {later}
    plans, Bs = zip(*(on_gpu(c, cuda, path="tensor_core", sort_rows=False) for c in cs))
    outs = [torch.full((c["M"], N), 5.0, dtype=torch.float32, device=cuda) for c in cs]
    f8 = precision == "e4m3"
    (tca_spmm.spmm_fp8_batched if f8 else tca_spmm.spmm_batched)(list(plans), list(Bs), outs, n_tile=n_tile)
    for p, C, c in zip(plans, outs, cs):
        p.status()
        ref = (oracle.spmm_fp8_f64 if f8 else oracle.spmm_f64)(c["row_ptr"], c["col"], c["vals"], c["B"])
        check(C, ref, c, False, f8)


@pytest.mark.parametrize("N", [256, 203])
@pytest.mark.parametrize("precision", ["f16", "e4m3"])
def test_popular_columns(cuda, N, precision):
    """4096 x 16384 with about 60 nonzeros a row, column k drawn in proportion
    to (k + 1)^-0.8: windows with a few chunks of popular columns (images, or
    consecutive columns) and tens of sparse ones, with the default options."""
    if precision == "e4m3" and N % 8:
        N = 208  # E4M3 takes multiples of 8
    rng = np.random.default_rng(5)
    K = 16384
    cdf = np.cumsum((np.arange(K) + 1.0) ** -0.8)
    draws = np.searchsorted(cdf / cdf[-1], rng.random((4096, 66)))
    c = csr([np.unique(d) for d in draws], K, rng, N)
    plan, B = on_gpu(c, cuda)
    if precision == "e4m3":
        C, ref = plan.spmm_fp8(B, out_dtype=torch.float16), oracle.spmm_fp8_f64(c["row_ptr"], c["col"], c["vals"], c["B"])
    else:
        C, ref = plan.spmm(B, out_dtype=torch.float16), oracle.spmm_f64(c["row_ptr"], c["col"], c["vals"], c["B"])
    plan.status()
    check(C, ref, c, True, precision == "e4m3")
