"""A batch whose bounds pass 8 GiB reads its sizes back first, in a head pass that has no room for cells and runs yet
and gathers the coordinates all the same.  Two jobs of 25 million points in one batch against each job alone, which
is laid out by bounds."""
import numpy as np
import pytest

import colo
from helpers import FIELDS

pytestmark = pytest.mark.gpu


def test_batch_past_the_bounds():
    n = 25_000_000
    ctx = colo.Context(0)
    box = np.array([0, 0, 6000, 6000], np.float32)
    dss = []
    for seed in (1, 2):
        rng = np.random.default_rng(seed)
        x, y = (rng.random(n, np.float32) * 6000 for _ in range(2))
        dss.append(colo.Dataset.from_arrays(ctx, x, y, np.repeat(np.arange(4, dtype=np.int32), n // 4), box))
    p = colo.default_params(0.5, 0.05, max_size=3)
    both = ctx.mine_batch(dss, [p, p])
    for ds, got in zip(dss, both):
        alone = ctx.mine(ds, p)
        assert len(got.levels) == len(alone.levels) >= 1 and got.levels[0].rows.any()
        for a, b in zip(alone.levels, got.levels):
            for f in FIELDS + ("pi",):
                assert np.array_equal(getattr(a, f), getattr(b, f)), (a.k, f)


def test_dataset_past_the_bounds():
    """One dataset of 50 million points alone (coordinates in id order, pairs over a queue) and beside a small one
    (coordinates gathered, pairs over every run); both read their sizes back first."""
    n = 50_000_000
    rng = np.random.default_rng(3)
    x, y = (rng.random(n, np.float32) * 9000 for _ in range(2))
    box = np.array([0, 0, 9000, 9000], np.float32)
    ctx = colo.Context(0)
    ds = colo.Dataset.from_arrays(ctx, x, y, np.repeat(np.arange(4, dtype=np.int32), n // 4), box)
    few = colo.Dataset.from_arrays(ctx, x[:50], y[:50], np.zeros(50, np.int32), box)
    p = colo.default_params(0.5, 0.05, max_size=3)
    alone, beside = ctx.mine(ds, p), ctx.mine_batch([ds, few], [p, p])[0]
    assert len(alone.levels) == len(beside.levels) >= 1 and alone.levels[0].rows.any()
    for a, b in zip(alone.levels, beside.levels):
        for f in FIELDS + ("pi",):
            assert np.array_equal(getattr(a, f), getattr(b, f)), (a.k, f)
