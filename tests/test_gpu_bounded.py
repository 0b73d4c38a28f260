"""Sizes that bucketing leaves on the device: everything up to the pairs' bounds is queued into arrays laid out
by bounds and read back with one wait.  Checked at the edges of the tiles (2048 points a head tile, 4096 a sort
tile), with no level to mine, with errors that are only seen at that wait, and when neighbours outgrow the room
of eight a point (the join runs again)."""
import numpy as np
import pytest

import colo
import oracle
from colo import gen
from colo.gen import Workload
from helpers import assert_same_trace, oracle_for, resolve_ambiguous

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return colo.Context(0)


def _uniform(n, features, width, seed):
    rng = np.random.default_rng(seed)
    fid = np.sort(rng.integers(0, features, n)).astype(np.int32)
    x, y = (rng.uniform(0, width, n).astype(np.float32) for _ in range(2))
    return Workload("uniform", x, y, fid, np.array([0, 0, width, width], np.float32), 10.0, 0.1, [], 3)


@pytest.mark.parametrize("n", [2, 255, 256, 257, 2047, 2048, 2049, 4095, 4096, 4097, 8193])
@pytest.mark.parametrize("width", [60.0, 2000.0])
def test_tile_edges(ctx, n, width):
    wl = _uniform(n, min(5, n), width, n)
    ds = colo.Dataset.from_arrays(ctx, wl.x, wl.y, wl.fid, wl.bounds)
    cell, rc, rf, rn = ctx.stage_cells(ds, wl.R)
    order = np.lexsort((wl.fid, cell))
    key = cell[order].astype(np.int64) * 16 + np.searchsorted(np.unique(wl.fid), wl.fid)[order]
    uniq, count = np.unique(key, return_counts=True)
    assert np.array_equal(rc.astype(np.int64) * 16 + rf, uniq) and np.array_equal(rn, count)
    for mode in (colo.MODE_BATCHED, colo.MODE_PLAIN):
        got = ctx.mine(ds, colo.default_params(wl.R, wl.thr, mode, max_size=wl.max_size))
        assert_same_trace(got, oracle_for(ctx, wl))


def test_neighbours_past_the_room(ctx):
    """700 points in one reach: 300 neighbours a point on average, far more than eight."""
    wl = _uniform(700, 6, 9.0, 5)
    wl.max_size = 2
    ds = colo.Dataset.from_arrays(ctx, wl.x, wl.y, wl.fid, wl.bounds)
    n = 14000   # 14,000 points: 9.8e7 capacity against a room of 1.8e5
    big = _uniform(n, 6, 60.0, 6)
    big.max_size = 2
    dsb = colo.Dataset.from_arrays(ctx, big.x, big.y, big.fid, big.bounds)
    for w, d in ((wl, ds), (big, dsb)):
        got = ctx.mine(d, colo.default_params(w.R, w.thr, colo.MODE_BATCHED, max_size=2))
        assert_same_trace(got, oracle_for(ctx, w))
        offs, nbr = ctx.stage_neighbors(d, w.R)
        o_offs, o_nbr, unres = oracle.neighbors(w.x, w.y, w.fid, w.bounds, w.R,
                                                res=resolve_ambiguous(ctx, w.x, w.y, w.fid, w.R))
        assert unres == 0 and np.array_equal(offs, o_offs) and np.array_equal(nbr, o_nbr)
        assert got.counters["neighbors"] == len(nbr)


def test_no_level_to_mine(ctx):
    """One feature: no pair, but the totals and the errors of bucketing are those of any mine."""
    wl = _uniform(3000, 1, 500.0, 9)
    ds = colo.Dataset.from_arrays(ctx, wl.x, wl.y, wl.fid, wl.bounds)
    got = ctx.mine(ds, colo.default_params(wl.R, wl.thr))
    assert got.levels == [] and got.counters["points"] == 3000 and got.counters["cells"] == got.counters["runs"] > 0
    y = wl.y.copy()
    y[17] = 5000.0
    ds = colo.Dataset.from_arrays(ctx, wl.x, y, wl.fid, wl.bounds)
    with pytest.raises(colo.ColoError) as e:
        ctx.mine(ds, colo.default_params(wl.R, wl.thr))
    assert e.value.status == colo.ERR_INPUT


def test_batch_with_an_empty_reach(ctx):
    """Jobs of one point, of one feature and of many in one batch."""
    jobs = [_uniform(1, 1, 100.0, 1), _uniform(2500, 7, 150.0, 2), _uniform(40, 1, 100.0, 3), gen.config(0)]
    dss = [colo.Dataset.from_arrays(ctx, w.x, w.y, w.fid, w.bounds) for w in jobs]
    ps = [colo.default_params(w.R, w.thr, colo.MODE_BATCHED, max_size=w.max_size) for w in jobs]
    for w, got in zip(jobs, ctx.mine_batch(dss, ps)):
        if w.nfeat < 2:
            assert got.levels == []
        else:
            assert_same_trace(got, oracle_for(ctx, w))
