"""Every layout that a size rule chooses, on small data: the device's memory that the rules see is lowered
(colo_params.reserved[2]), so that a few thousand points are laid out by bounds, with the head arrays for every point, or
with the heads counted first (a launch without room, then one with), with the sort's look-back words for all passes or
one pass's, and joined in a single pass, in one made again with room, or in count + scan + fill.  Which of them ran is
read from the profiled pass; traces and tables (whose row order is the neighbour lists' order) are the oracle's."""
import numpy as np
import pytest

import colo
from colo.gen import Workload
from helpers import FIELDS, assert_same_trace, oracle_for

pytestmark = pytest.mark.gpu

# the device's memory in KiB: its 16th holds all bounds, the heads of every point, not even those (for 20,000 points)
BOUNDS, HEADS, COUNTED = 98304, 32768, 4096


@pytest.fixture(scope="module")
def ctx():
    return colo.Context(0)


def _points(n, features, width, lines, seed):
    """Half the points uniform, half around the crossings of `lines` columns and rows (the fewer, the longer the lists)."""
    rng = np.random.default_rng(seed)
    at = rng.uniform(0.1 * width, 0.9 * width, (2, lines))
    x, y = (np.where(np.arange(n) % 2, rng.uniform(0, width, n),
                     np.clip(rng.choice(a, n) + rng.normal(0, 6, n), 0, width)).astype(np.float32) for a in at)
    fid = np.sort(rng.integers(0, features, n)).astype(np.int32)
    return Workload("layouts", x, y, fid, np.array([0, 0, width, width], np.float32), 10.0, 0.2, [], 3)


def _params(wl, kib, mode=colo.MODE_BATCHED):
    p = colo.default_params(wl.R, wl.thr, mode, max_size=wl.max_size, keep_tables=True, profile=True)
    p.reserved[2] = kib
    return p


def _layout(got):
    k = got.kernels
    if "host cell_heads" in k:
        assert k["cell_heads"][0] == 2
        return COUNTED
    assert k["cell_heads"][0] == 1
    return HEADS if "host cell_masks" in k else BOUNDS


def _form(got):
    assert ("join_count" in got.kernels) == ("join_fill" in got.kernels)
    if "join_fill" in got.kernels:
        return "two passes"
    return "again" if got.kernels["join"][0] == 2 else "single"


# lines for 20,000 points: about 110,000 pairs, 290,000 (above the room of eight a point) and 500,000 (above every cap)
DENSITY = {"few": 20, "some": 12, "many": 9}


@pytest.mark.parametrize("kib", [BOUNDS, HEADS, COUNTED])
@pytest.mark.parametrize("density", DENSITY)
@pytest.mark.parametrize("width", [1, 8, 32])
def test_one_job(ctx, kib, density, width):
    wl = _points(20000, 6, 6000.0, DENSITY[density], 7)
    ds = colo.Dataset.from_arrays(ctx, wl.x, wl.y, wl.fid, wl.bounds)
    ctx.set_join_group(width)
    try:
        got = ctx.mine(ds, _params(wl, kib))
    finally:
        ctx.set_join_group(0)
    assert _layout(got) == kib
    pairs, cap = got.counters["join_pairs"], kib * 4
    room = min(cap, 8 * 20000 + 65536) if kib == BOUNDS else 0
    assert _form(got) == ("two passes" if pairs > cap else "again" if kib == BOUNDS and pairs > room else "single")
    assert_same_trace(got, oracle_for(ctx, wl, keep_tables=True), tables=True)


def test_the_cases_reach_every_form(ctx):
    forms = {}
    for kib in (BOUNDS, HEADS, COUNTED):
        for density, lines in DENSITY.items():
            wl = _points(20000, 6, 6000.0, lines, 7)
            ds = colo.Dataset.from_arrays(ctx, wl.x, wl.y, wl.fid, wl.bounds)
            forms[kib, density] = _form(ctx.mine(ds, _params(wl, kib)))
    assert [forms[BOUNDS, d] for d in DENSITY] == ["single", "again", "two passes"], forms
    assert [forms[HEADS, d] for d in DENSITY] == ["single", "two passes", "two passes"], forms
    assert [forms[COUNTED, d] for d in DENSITY] == ["two passes"] * 3, forms


@pytest.mark.parametrize("kib", [BOUNDS, HEADS, COUNTED])
@pytest.mark.parametrize("lines", [12, 7, 4])
def test_several_jobs(ctx, kib, lines):
    jobs = [_points(n, f, 6000.0, lines, s) for n, f, s in ((9000, 5, 1), (40, 3, 2), (11000, 40, 3))]
    jobs[2].thr = 0.02
    dss = [colo.Dataset.from_arrays(ctx, w.x, w.y, w.fid, w.bounds) for w in jobs]
    got = ctx.mine_batch(dss, [_params(w, kib) for w in jobs])
    assert _layout(got[0]) == kib
    first = 0   # a batched job's tables number the points of the whole batch
    for w, r in zip(jobs, got):
        for lev in r.levels:
            lev.tables = {c: t - np.uint32(first) for c, t in lev.tables.items()}
        assert_same_trace(r, oracle_for(ctx, w, keep_tables=True), tables=True)
        first += w.n


@pytest.mark.parametrize("box", [600.0, 4000.0, 40000.0, 1e6])   # 12, 18, 24 and 34 key bits
@pytest.mark.parametrize("n", [2, 4097, 30011])
def test_sort_words_of_one_pass(ctx, n, box):
    wl = _points(n, 2, box, 200, n)
    ds = colo.Dataset.from_arrays(ctx, wl.x, wl.y, wl.fid, wl.bounds)
    got = ctx.mine(ds, _params(wl, 1))
    assert_same_trace(got, oracle_for(ctx, wl, keep_tables=True), tables=True)


def test_ids_instead_of_gathered_coordinates(ctx):
    """Above 2^23 points the lists hold ids; heads counted first and pairs in two passes against the default layout."""
    n = (1 << 23) + 5
    rng = np.random.default_rng(11)
    x, y = (rng.random(n, np.float32) * 4000 for _ in range(2))
    fid = np.sort(rng.integers(0, 5, n)).astype(np.int32)
    ds = colo.Dataset.from_arrays(ctx, x, y, fid, np.array([0, 0, 4000, 4000], np.float32))
    a, b = (colo.default_params(0.9, 0.01, max_size=3, profile=True) for _ in range(2))
    b.reserved[2] = 65536
    a, b = ctx.mine(ds, a), ctx.mine(ds, b)
    assert _layout(a) == BOUNDS and _layout(b) == COUNTED and _form(b) == "two passes"
    assert len(a.levels) == len(b.levels) >= 2 and a.levels[0].rows.any()
    for p, q in zip(a.levels, b.levels):
        for f in FIELDS + ("pi",):
            assert np.array_equal(getattr(p, f), getattr(q, f)), (p.k, f)
