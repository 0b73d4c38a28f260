"""The level filter looks only at cells with a quad of three features or more (fewer when a pattern names a feature
more than once): bounds against a brute-force count over the quads, for grids with few and with many such cells, at
the grid's edges, with none at all, and for several jobs in one batch whose cells share warps."""
import itertools

import numpy as np
import pytest

import colo
from colo import gen
from helpers import assert_same_trace, oracle_for

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return colo.Context(0)


def _bounds(x, y, fid, gx, gy, cand):
    """Sum over the cells of full quads of each member's points (unit cells, lower corner 0, 0)."""
    cnt = np.zeros((gy, gx, fid.max() + 1), np.int64)
    np.add.at(cnt, (y.astype(int), x.astype(int), fid), 1)
    out = []
    for c in cand:
        u = np.zeros((gy, gx), bool)
        for by, bx in itertools.product(range(gy - 1), range(gx - 1)):
            q = cnt[by:by + 2, bx:bx + 2]
            if all(q[..., f].any() for f in c):
                u[by:by + 2, bx:bx + 2] = True
        out.append([cnt[u][:, f].sum() for f in c])
    return np.array(out)


@pytest.mark.parametrize("n,side,features", [(40, 12, 3), (90, 12, 4), (400, 20, 5), (1500, 20, 6), (60, 40, 5), (300, 3, 3)])
def test_bounds(ctx, n, side, features):
    rng = np.random.default_rng(n + side)
    x, y = (rng.uniform(0, side, n).astype(np.float32) for _ in range(2))
    fid = np.sort(np.r_[np.arange(features), rng.integers(0, features, n - features)]).astype(np.int32)
    # the grid has a row more than the bounds' height (its upper edge is bounds + distance)
    ds = colo.Dataset.from_arrays(ctx, x, y, fid, np.array([0, 0, side, side], np.float32))
    for cand in (list(itertools.combinations(range(features), 3)),
                 [(0, 0, 1), (1, 1, 1), (0, 1, 2)],
                 [(2, 2, 2)]):
        ub, _ = ctx.stage_filter(ds, 1.0, 0.1, np.array(cand, np.uint32))
        assert np.array_equal(ub.astype(np.int64), _bounds(x, y, fid, side, side + 1, cand)), cand


def test_no_such_cell(ctx):
    """Every cell of its own feature, two apart: no quad holds two."""
    g = np.arange(10, dtype=np.float32) * 3 + 0.5
    x, y = (v.ravel() for v in np.meshgrid(g, g))
    fid = np.sort(np.arange(100) % 5).astype(np.int32)
    ds = colo.Dataset.from_arrays(ctx, x, y, fid, np.array([0, 0, 30, 30], np.float32))
    ub, ok = ctx.stage_filter(ds, 1.0, 0.1, np.array([(0, 1, 2), (2, 3, 4)], np.uint32))
    assert not ub.any() and not ok.any()
    res = ctx.mine(ds, colo.default_params(1.0, 0.0, max_size=4))   # everything passes at 0
    assert [len(lev.cand) for lev in res.levels] == [10, 10, 5] and not any(lev.ub.any() for lev in res.levels)


@pytest.mark.parametrize("jobs", [2, 9, 40])
def test_jobs_that_share_warps(ctx, jobs):
    """Jobs of a few cells each: a warp of the queue holds cells of several."""
    wls = [gen.config(0, seed=s) for s in range(jobs)]
    for s, w in enumerate(wls):
        keep = np.arange(w.n) % (1 + s % 4) == 0
        w.x, w.y, w.fid = w.x[keep], w.y[keep], w.fid[keep]
    dss = [colo.Dataset.from_arrays(ctx, w.x, w.y, w.fid, w.bounds) for w in wls]
    got = ctx.mine_batch(dss, [colo.default_params(w.R, w.thr, max_size=w.max_size) for w in wls])
    for w, r in zip(wls, got):
        assert_same_trace(r, oracle_for(ctx, w))


@pytest.mark.parametrize("n", [(1 << 21) - 1, 1 << 21])
@pytest.mark.parametrize("features", [6, 300])
def test_pairs_on_both_sides_of_the_queue(ctx, n, features):
    """From 2^21 points on a single job's pairs are bounded over a queue of cells, else over every run (as beside a
    second job): the same bounds, with block-private sums and without, and a spot of cells with many runs."""
    rng = np.random.default_rng(n + features)
    x, y = (rng.random(n, np.float32) * 2000 for _ in range(2))
    fid = np.sort(rng.integers(0, features, n, np.int32))
    spot = rng.choice(n, 4000, replace=False)
    x[spot], y[spot] = (rng.normal(700, 1.5, 4000).astype(np.float32) for _ in range(2))
    box = np.array([0, 0, 2000, 2000], np.float32)
    ds = colo.Dataset.from_arrays(ctx, x, y, fid, box)
    few = colo.Dataset.from_arrays(ctx, x[:50], y[:50], np.zeros(50, np.int32), box)
    p = colo.default_params(0.5, 0.9, max_size=2)
    alone, beside = ctx.mine(ds, p), ctx.mine_batch([ds, few], [p, p])[0]
    assert len(alone.levels) == 1 and alone.levels[0].ub.any()
    for f in ("cand", "ub", "passed", "rows", "num", "pi"):
        assert np.array_equal(getattr(alone.levels[0], f), getattr(beside.levels[0], f)), f


@pytest.mark.parametrize("features", [79, 80, 81, 113, 114, 160, 161, 226, 227])
def test_pair_block_sizes(ctx, features):
    """Feature counts on both sides of every block size that the accumulator allows, and past it."""
    rng = np.random.default_rng(features)
    n = 6000
    x, y = (rng.uniform(0, 40, n).astype(np.float32) for _ in range(2))
    fid = np.sort(np.r_[np.arange(features), rng.integers(0, features, n - features)]).astype(np.int32)
    ds = colo.Dataset.from_arrays(ctx, x, y, fid, np.array([0, 0, 40, 40], np.float32))
    cand = rng.choice(features, (40, 2), replace=True)
    cand = np.sort(cand[cand[:, 0] != cand[:, 1]], axis=1)
    ub, _ = ctx.stage_filter(ds, 1.0, 0.1, cand.astype(np.uint32))
    assert np.array_equal(ub.astype(np.int64), _bounds(x, y, fid, 40, 41, cand))
