"""The sort over every split of a key into digits (passes of eight bits, of nine where that saves a pass, 32- and
64-bit keys), and the cells and runs found after it for feature counts around powers of two."""
import numpy as np
import pytest

import colo

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return colo.Context(0)


def _check(ctx, x, y, fid, box, R):
    ds = colo.Dataset.from_arrays(ctx, x, y, fid, box)
    cell, rc, rf, rn = ctx.stage_cells(ds, R)
    key = np.stack([cell, np.searchsorted(np.unique(fid), fid).astype(np.uint64)], axis=1)
    uniq, count = np.unique(key, axis=0, return_counts=True)
    assert np.array_equal(rc, uniq[:, 0]) and np.array_equal(rf, uniq[:, 1]) and np.array_equal(rn, count)
    return ds, cell


@pytest.mark.parametrize("n", [3000, 30001])
@pytest.mark.parametrize("bits", list(range(2, 41)))
def test_digit_splits(ctx, bits, n):
    rng = np.random.default_rng(bits)
    w, h = float(2 ** (bits // 2)), float(2 ** (bits - bits // 2))
    x, y = rng.uniform(0, w, n).astype(np.float32), rng.uniform(0, h, n).astype(np.float32)
    # half of the points in a corner of the grid: cells of many points at every width
    x[::2] = np.minimum(x[::2], rng.uniform(0, 8, (n + 1) // 2).astype(np.float32))
    y[::2] = np.minimum(y[::2], rng.uniform(0, 8, (n + 1) // 2).astype(np.float32))
    fid = np.sort(rng.integers(0, 7, n)).astype(np.int32)
    ds, cell = _check(ctx, x, y, fid, np.array([0, 0, w, h], np.float32), 1.0)
    if n == 3000 and bits >= 6:
        # a stable sort: within a cell and a feature the points ascend
        off, nb = ctx.stage_neighbors(ds, 1.0)
        for a in np.nonzero(np.diff(off.astype(np.int64)) > 1)[0][:200]:
            lst = nb[int(off[a]):int(off[a + 1])]
            order = np.lexsort((lst, cell[lst], fid[lst]))
            assert np.array_equal(order, np.arange(len(lst)))


@pytest.mark.parametrize("features", [1, 2, 3, 4, 5, 31, 32, 33, 64, 65, 127, 128, 129])
def test_feature_counts(ctx, features):
    n = 2048 * 3 + 77
    rng = np.random.default_rng(features)
    fid = np.sort(rng.integers(0, features, n) ** 2 // max(features, 1)).astype(np.int32)   # few points in high features
    x, y = (rng.uniform(0, 40, n).astype(np.float32) for _ in range(2))
    _check(ctx, x, y, fid, np.array([0, 0, 40, 40], np.float32), 1.0)
