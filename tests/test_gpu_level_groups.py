"""Candidates that share a parent table are counted together, up to 32 extensions at a time.  Groups of one, of
more than one, of exactly 32 and of more (split), rows on both sides of a 32-row chunk, and rows whose lists hold
features that are no extension, against the oracle: every field and every table in row order, in all forms."""
import numpy as np
import pytest

import colo
from colo.gen import Workload
from helpers import assert_same_trace, oracle_for

pytestmark = pytest.mark.gpu


def _cliques(features, rows, per, seed, width):
    """`rows` clusters with `per` points of every feature within one reach, far from each other, and two
    scattered points of every feature."""
    rng = np.random.default_rng(seed)
    cx, cy = 60.0 + 100.0 * np.arange(rows), np.full(rows, 50.0)
    x = np.concatenate([np.concatenate([np.repeat(cx, per) + rng.uniform(-3, 3, rows * per), rng.uniform(0, width, 2)])
                        for _ in range(features)])
    y = np.concatenate([np.concatenate([np.repeat(cy, per) + rng.uniform(-3, 3, rows * per), rng.uniform(0, 100, 2)])
                        for _ in range(features)])
    return x.astype(np.float32), y.astype(np.float32), np.repeat(np.arange(features, dtype=np.int32), rows * per + 2)


@pytest.mark.parametrize("features,rows,per,max_size", [
    (3, 1, 1, 0), (3, 31, 1, 0), (4, 32, 1, 0), (4, 33, 2, 0), (33, 3, 1, 3), (34, 5, 1, 3), (70, 2, 1, 3), (6, 40, 3, 5),
    (10, 3, 1, 0)])
def test_groups_match_the_oracle(features, rows, per, max_size):
    width = 100.0 * rows + 100.0
    x, y, fid = _cliques(features, rows, per, features * 10 + rows, width)
    wl = Workload("cliques", x, y, fid, np.array([0, 0, width, 100], np.float32), 12.0, 0.05, [], max_size)
    ctx = colo.Context(0)
    ds = colo.Dataset.from_arrays(ctx, wl.x, wl.y, wl.fid, wl.bounds)
    ref = oracle_for(ctx, wl, keep_tables=True)
    assert len(ref.levels) > 1
    for mode in (colo.MODE_BATCHED, colo.MODE_PLAIN):
        got = ctx.mine(ds, colo.default_params(wl.R, wl.thr, mode, max_size=max_size, keep_tables=True))
        assert_same_trace(got, ref, tables=True)
    for queue in (0, 1):
        ctx.set_tuning(level_block=64, level_queue=queue)
        got = ctx.mine(ds, colo.default_params(wl.R, wl.thr, colo.MODE_BATCHED, max_size=max_size, keep_tables=True))
        assert_same_trace(got, ref, tables=True)
