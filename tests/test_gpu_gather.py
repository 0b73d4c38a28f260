"""Above 2^23 points a single dataset's lists and anchors name points by id and the join reads the coordinates in id
order; up to there, and for several jobs, they are gathered into cell order first.  Both give the same levels and
tables: one dataset on either side of the line alone and beside a second one, with a dense spot for the long lists."""
import numpy as np
import pytest

import colo
from helpers import FIELDS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1 << 23, (1 << 23) + 1])
def test_alone_and_in_a_batch(n):
    rng = np.random.default_rng(n)
    x, y = (rng.random(n, np.float32) * 4000 for _ in range(2))
    fid = np.sort(rng.integers(0, 6, n, np.int32))
    spot = rng.choice(n, 3000, replace=False)
    x[spot], y[spot] = (rng.normal(700, 1.5, 3000).astype(np.float32) for _ in range(2))
    ctx = colo.Context(0)
    box = np.array([0, 0, 4000, 4000], np.float32)
    ds = colo.Dataset.from_arrays(ctx, x, y, fid, box)
    few = colo.Dataset.from_arrays(ctx, x[:50], y[:50], np.zeros(50, np.int32), box)
    p = colo.default_params(1.0, 0.2, max_size=3, keep_tables=True)
    alone = ctx.mine(ds, p)
    beside = ctx.mine_batch([ds, few], [p, p])[0]
    assert len(alone.levels) == len(beside.levels) == 2 and alone.counters["neighbors"] > n // 2
    for a, b in zip(alone.levels, beside.levels):
        for f in FIELDS + ("pi",):
            assert np.array_equal(getattr(a, f), getattr(b, f)), (a.k, f)
        assert (a.tables or a.k > 2) and a.tables.keys() == b.tables.keys()
        for c, t in a.tables.items():
            assert np.array_equal(t, b.tables[c])
