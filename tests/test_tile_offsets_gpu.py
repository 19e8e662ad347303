"""The chunk offsets of a plan around the chunk count from which a library scan
makes them (512): against the host build, array by array."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import tca_spmm  # noqa: E402


@pytest.mark.parametrize("windows,blocks", [(1, 1), (7, 73), (8, 64), (9, 57), (30, 70)])  # 1, 511, 512, 513, 2100 chunks
def test_tile_offsets(cuda, windows, blocks):
    rng = np.random.default_rng(windows)
    M, K = 128 * windows - 3, 64 * blocks
    rows = [np.sort(rng.choice(K, max(1, K // 25), replace=False)) for _ in range(M)]
    row_ptr = np.concatenate([[0], np.cumsum([r.size for r in rows])]).astype(np.int32)
    col = np.concatenate(rows).astype(np.int32)
    vals = rng.standard_normal(col.size).astype(np.float16)
    want = oracle.build_plan(row_ptr, col, vals, K, path=2)
    assert want["n_tc_chunks"] == windows * blocks
    plan = tca_spmm.Plan(*(torch.from_numpy(x).to(cuda) for x in (row_ptr, col, vals)), K, path="tensor_core")
    for which, name in ((tca_spmm.ARR_TILE_PTR, "tile_ptr"), (tca_spmm.ARR_WIN_COLS, "win_cols"),
                        (tca_spmm.ARR_TILE_SRC, "tile_src")):
        assert np.array_equal(plan.export(which), want[name])
    got = plan.export(tca_spmm.ARR_TILE_ENTRIES)
    assert np.array_equal(got[:want["tile_entries"].size], want["tile_entries"])
