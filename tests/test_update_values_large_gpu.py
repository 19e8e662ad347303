"""New values for plans of many chunks: thousands of sparse chunks with some
images among them (entries walked without their chunks), and more images than
are cut into parts -- arrays equal to those of a plan built from the values, bit
for bit, the transpose's forward too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import tca_spmm  # noqa: E402


@pytest.mark.parametrize("M,K,spread,front", [(8190, 8192, 80, 30), (8192, 8150, 60, 0), (4096, 1024, 130, 0), (4000, 1000, 20, 12)])
def test_update_matches_fresh_plan(cuda, M, K, spread, front):
    rng = np.random.default_rng(M + spread)
    step = K // spread  # `spread` columns all over K, `front` among the first 64
    rows = []
    for _ in range(M):
        r = np.arange(spread) * step + rng.integers(0, step, spread)
        rows.append(np.union1d(r, rng.choice(64, front, replace=False)) if front else r)
    row_ptr = np.concatenate([[0], np.cumsum([r.size for r in rows])]).astype(np.int32)
    col = np.concatenate(rows).astype(np.int32)
    rp, ci = torch.from_numpy(row_ptr).to(cuda), torch.from_numpy(col).to(cuda)
    v, new = (torch.from_numpy(rng.standard_normal(col.size).astype(np.float16)).to(cuda) for _ in range(2))
    plan = tca_spmm.Plan(rp, ci, v, K, path="tensor_core")
    plan.build_transpose()
    plan.update_values(new)
    fresh = tca_spmm.Plan(rp, ci, new, K, path="tensor_core")
    for which in (tca_spmm.ARR_P_VAL, tca_spmm.ARR_TILE_ENTRIES, tca_spmm.ARR_TILE_IMAGES):
        assert np.array_equal(plan.export(which), fresh.export(which))
    dY = torch.randn((M, 64), device=cuda).half()
    assert torch.equal(plan.spmm_t(dY), fresh.spmm_t(dY))
