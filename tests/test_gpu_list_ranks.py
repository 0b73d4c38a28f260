"""Cells with long neighbourhood lists are merged by a warp from the ranks of features in its neighbours' masks: every
mask width around a multiple of 32 features and the padded ones, several such cells per warp, lists with and without
each feature in every neighbour, against brute force.  Coordinates and distance are exact in binary."""
import numpy as np
import pytest

import colo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("features", [1, 2, 31, 32, 33, 64, 65, 127, 256, 257, 384, 385, 700, 1024])
@pytest.mark.parametrize("side", [2, 5])
def test_long_lists_by_rank(features, side):
    ctx = colo.Context(0)
    rng = np.random.default_rng(features)
    n = max(2200, features)
    fid = np.sort(np.r_[np.arange(features), rng.integers(0, features, n - features)]).astype(np.int32)
    x, y = (((rng.integers(0, 8 * side, n) + 16) / 8).astype(np.float32) for _ in range(2))
    box = np.array([0, 0, 12, 12], np.float32)
    ds = colo.Dataset.from_arrays(ctx, x, y, fid, box)
    off, nb = ctx.stage_neighbors(ds, 1.0)
    cell = ctx.stage_cells(ds, 1.0)[0]
    d2 = (x[:, None].astype(np.float64) - x) ** 2 + (y[:, None].astype(np.float64) - y) ** 2
    near = (d2 <= 1.0) & (fid[None, :] > fid[:, None])
    order = np.lexsort((np.arange(n), cell, fid))
    assert int(off[-1]) == int(near.sum())
    for a in range(n):
        want = order[near[a][order]]
        assert np.array_equal(nb[int(off[a]):int(off[a + 1])], want), a
