"""A level of three or more members is filtered and counted with one wait, the candidates' bounds being tested in
the count kernel against the least bound that passes; a mine that records features waits for the filter first.
Both give the same levels, at thresholds that ratios of the data reach exactly, at 0 and 1, and with parent tables
on both sides of the 16,384 rows up to which a learned mine takes one wait."""
import numpy as np
import pytest

import colo
from colo import gen
from helpers import FIELDS, assert_same_trace, oracle_for

pytestmark = pytest.mark.gpu


def _same(a, b):
    assert len(a.levels) == len(b.levels)
    for x, y in zip(a.levels, b.levels):
        for f in FIELDS + ("pi",):
            assert np.array_equal(getattr(x, f), getattr(y, f)), (x.k, f)
    for c in ("filter_cells", "filter_full_quads", "refined", "count_items", "count_parent_words", "bitmap_words"):
        assert a.counters[c] == b.counters[c], c


@pytest.mark.parametrize("thr", [0.0, 1.0, 0.2, 0.1, 0.05])
def test_one_wait_matches_two(thr):
    ctx = colo.Context(0)
    wl = gen.config(1, scale=0.02)
    wl.max_size = 4
    ds = colo.Dataset.from_arrays(ctx, wl.x, wl.y, wl.fid, wl.bounds)
    thrs = [thr]
    if thr == 0.1:   # ratios that occur: a level-3 candidate's smallest bound over its feature's instances
        base = ctx.mine(ds, colo.default_params(wl.R, 0.02, max_size=3))
        n = np.bincount(wl.fid)
        for lev in base.levels[1:]:
            for c in range(0, len(lev.cand), max(1, len(lev.cand) // 6)):
                r = np.float32(np.min(lev.ub[c] / n[lev.cand[c]].astype(np.float64)))
                thrs += [float(r), float(np.nextafter(r, np.float32(2)))]
    for t in thrs:
        if t == 0.0:   # everything passes: every triple of 40 features
            wl.max_size = 3
        one = ctx.mine(ds, colo.default_params(wl.R, t, max_size=wl.max_size))
        two = ctx.mine(ds, colo.default_params(wl.R, t, max_size=wl.max_size, features=True))
        _same(one, two)
        wl.thr = t
        if t >= 0.05:
            assert_same_trace(one, oracle_for(ctx, wl))


@pytest.mark.parametrize("scale", [0.02, 0.3])
def test_learned_parent_lengths(scale):
    ctx = colo.Context(0)
    ctx.set_model(colo.load_model())
    wl = gen.config(3, scale=scale)
    ds = colo.Dataset.from_arrays(ctx, wl.x, wl.y, wl.fid, wl.bounds)
    a = ctx.mine(ds, colo.default_params(wl.R, wl.thr, colo.MODE_LEARNED))
    longest = max(int(lev.rows[lev.prevalent.astype(bool)].max(initial=0)) for lev in a.levels)
    assert (longest > 16384) == (scale > 0.1)
    _same(a, ctx.mine(ds, colo.default_params(wl.R, wl.thr, colo.MODE_BATCHED)))
    _same(a, ctx.mine(ds, colo.default_params(wl.R, wl.thr, colo.MODE_LEARNED, features=True)))
