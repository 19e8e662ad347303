"""The tensor-core kernel's stage ring at the edges of its batches: chunk
streams shorter than the ring, of one batch of chunk records (28 and 32
chunks) and one more, and of several; image, sparse and condensed chunks in
one launch; N of whole 64-column slabs (one 3-D box per chunk) and not (a 2-D
box per slab); beta = 0 (coalesced stores) and beta != 0.

Tolerance, elementwise: the FP16 products are exact in FP32 (E4M3 ones too),
so |error| <= n_r 2^-23 (|A| |B|)[r, n] for a row of n_r nonzeros accumulated
in FP32 in any order, plus 2^-11 |ref| + 2^-24 for FP16 output and, with E4M3,
2^-21 |ref| for the two scale products."""
import numpy as np
import pytest

from oracle import oracle
from tca_spmm import gen

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import tca_spmm  # noqa: E402


def matrix(chunks, N, seed):
    """Three windows over `chunks` 64-column blocks (the last one ragged):
    rows dense enough for tile images, sparse rows, and rows that only use 70
    scattered columns (condensed: gathered B rows)."""
    rng = np.random.default_rng(seed)
    K = max(chunks * 64 - 5, 70)
    mask = np.zeros((128 * 3 - 7, K), bool)
    mask[:128] = rng.random((128, K)) < 0.25
    mask[128:256] = rng.random((128, K)) < 0.03
    few = np.sort(rng.choice(K, 70, replace=False))
    mask[256:, few] = rng.random((mask.shape[0] - 256, 70)) < 0.4
    row_nnz = mask.sum(1)
    row_ptr = np.concatenate([[0], np.cumsum(row_nnz)]).astype(np.int32)
    col = np.nonzero(mask)[1].astype(np.int32)
    vals = (rng.standard_normal(col.size) * 0.1).astype(np.float16)
    return dict(M=mask.shape[0], K=K, N=N, row_ptr=row_ptr, col=col, vals=vals, B=gen.uniform_b(rng, K, N))


def check(got, ref, c, f16, extra=0.0, vals=None, B=None):
    n_r = np.diff(c["row_ptr"])[:, None]
    mag = oracle.spmm_f64(c["row_ptr"], c["col"], np.abs(c["vals"]) if vals is None else vals,
                          np.abs(c["B"]) if B is None else B)
    tol = n_r * 2.0 ** -23 * mag + extra * np.abs(ref)
    if f16:
        tol = tol + 2.0 ** -11 * np.abs(ref) + 2.0 ** -24
    assert np.all(np.abs(got.cpu().numpy().astype(np.float64) - ref) <= tol)


SHAPES = [(1, 64), (2, 8), (4, 256), (5, 72), (28, 128), (29, 64), (32, 264), (33, 256), (61, 136), (65, 200)]


@pytest.mark.parametrize("chunks,N", SHAPES)
@pytest.mark.parametrize("out", ["f16", "f32"])
@pytest.mark.parametrize("n_tile", [64, 256])
def test_ring_f16(cuda, chunks, N, out, n_tile):
    c = matrix(chunks, N, 31 * chunks + N)
    dev = [torch.from_numpy(c[k]).to(cuda) for k in ("row_ptr", "col", "vals", "B")]
    plan = tca_spmm.Plan(*dev[:3], c["K"], path="tensor_core")
    C = torch.full((c["M"], N), 7.0, dtype=torch.float16 if out == "f16" else torch.float32, device=cuda)
    tca_spmm.spmm_batched([plan], [dev[3]], [C], n_tile=n_tile)
    plan.status()
    ref = oracle.spmm_f64(c["row_ptr"], c["col"], c["vals"], c["B"])
    check(C, ref, c, out == "f16")
    old = torch.full_like(C, 0.5)
    tca_spmm.spmm_batched([plan], [dev[3]], [old], alpha=2.0, beta=1.0, n_tile=n_tile)
    plan.status()
    # alpha doubles the sum's error; beta * C is exact, its addition rounds once more (2^-24)
    check(old / 2, ref + 0.25, c, out == "f16", extra=2.0 ** -23)


@pytest.mark.parametrize("chunks,N", SHAPES)
@pytest.mark.parametrize("out", ["f16", "f32"])
def test_ring_e4m3(cuda, chunks, N, out):
    c = matrix(chunks, N, 57 * chunks + N)
    dev = [torch.from_numpy(c[k]).to(cuda) for k in ("row_ptr", "col", "vals", "B")]
    plan = tca_spmm.Plan(*dev[:3], c["K"], path="tensor_core")
    C = plan.spmm_fp8(dev[3], out_dtype=torch.float16 if out == "f16" else torch.float32)
    plan.status()
    ref = oracle.spmm_fp8_f64(c["row_ptr"], c["col"], c["vals"], c["B"])
    # the quantized operands' magnitudes exceed the FP16 ones by at most 2^-4 each
    check(C, ref, c, out == "f16", extra=2.0 ** -21, vals=np.abs(c["vals"]) * np.float16(1.0625),
          B=np.abs(c["B"]) * np.float16(1.0625))


@pytest.mark.parametrize("precision", ["f16", "e4m3"])
@pytest.mark.parametrize("n_tile", [0, 128])
def test_mixed_widths_one_launch(cuda, precision, n_tile):
    """Jobs of different N-slice widths, chunk counts and N (whole slabs and
    not) in one launch; more jobs than one launch holds."""
    specs = [(3, 64), (17, 8), (1, 256), (9, 136), (5, 520), (33, 200), (2, 128)] * 5
    cs = [matrix(ch, N, 7 * i + N) for i, (ch, N) in enumerate(specs)]
    plans, Bs, outs = [], [], []
    for c in cs:
        rp, ci, v, B = (torch.from_numpy(c[k]).to(cuda) for k in ("row_ptr", "col", "vals", "B"))
        plans.append(tca_spmm.Plan(rp, ci, v, c["K"], path="tensor_core"))
        Bs.append(B)
        outs.append(torch.full((c["M"], c["N"]), 5.0, dtype=torch.float32, device=cuda))
    f8 = precision == "e4m3"
    (tca_spmm.spmm_fp8_batched if f8 else tca_spmm.spmm_batched)(plans, Bs, outs, n_tile=n_tile)
    for p, C, c in zip(plans, outs, cs):
        p.status()
        if f8:
            check(C, oracle.spmm_fp8_f64(c["row_ptr"], c["col"], c["vals"], c["B"]), c, False, extra=2.0 ** -21,
                  vals=np.abs(c["vals"]) * np.float16(1.0625), B=np.abs(c["B"]) * np.float16(1.0625))
        else:
            check(C, oracle.spmm_f64(c["row_ptr"], c["col"], c["vals"], c["B"]), c, False)
