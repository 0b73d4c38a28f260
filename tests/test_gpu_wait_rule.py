"""Which levels are filtered and counted with one wait: level 3 with few candidates, short tables and small features, a
later one when the filter passed nearly all of the last.  Features that meet pairwise in different places make every
pair prevalent and every triple stopped by the filter; groups of features that meet in one place make patterns that
all pass.  The waits are those of the profiled pass; the levels are the oracle's on both sides of each bound."""
import numpy as np
import pytest

import colo
from colo.gen import Workload
from helpers import assert_same_trace, oracle_for

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return colo.Context(0)


def _places(groups, each, copies=1, seed=1):
    """`each` places per group of features, `copies` points of each of its features in every one of them."""
    rng = np.random.default_rng(seed)
    at = [(g, i) for i, g in enumerate(g for g in groups for _ in range(each))]
    side = int(np.ceil(np.sqrt(len(at))))
    f, p = (np.array(v) for v in zip(*[(f, i) for g, i in at for f in g for _ in range(copies)]))
    x, y = (4.0 * (p % side) + 2, 4.0 * (p // side) + 2)
    x, y = (v + rng.uniform(-0.2, 0.2, len(p)) for v in (x, y))
    o = np.argsort(f, kind="stable")
    box = np.array([0, 0, 4.0 * side, 4.0 * side], np.float32)
    return Workload("places", x[o].astype(np.float32), y[o].astype(np.float32), f[o].astype(np.int32), box, 1.0, 0.0, [], 5)


def _waits(ctx, wl):
    """Levels past the pairs, and how many of them waited for the filter first."""
    ds = colo.Dataset.from_arrays(ctx, wl.x, wl.y, wl.fid, wl.bounds)
    got = ctx.mine(ds, colo.default_params(wl.R, wl.thr, max_size=wl.max_size, profile=True))
    assert_same_trace(got, oracle_for(ctx, wl))
    return got, got.kernels.get("part filter wait", (0, 0.0))[0]


def _pairs(F):
    return [(a, b) for a in range(F) for b in range(a + 1, F)]


# 12 features: 220 triples, 13: 286; past 2^17 chunks of 32 rows of triples' parents; past 2^21 words
@pytest.mark.parametrize("F,each,copies,two", [(3, 3, 1, False), (12, 3, 1, False), (13, 3, 1, True), (12, 74, 16, False),
                                               (12, 80, 16, True)])
def test_triples_that_the_filter_stops(ctx, F, each, copies, two):
    wl = _places(_pairs(F), each, copies)
    wl.thr = 0.5 / (F - 1)
    got, waits = _waits(ctx, wl)
    assert [lev.k for lev in got.levels] == [2, 3] and got.levels[0].prevalent.all() and not got.levels[1].passed.any()
    assert len(got.levels[1].cand) == F * (F - 1) * (F - 2) // 6
    chunks = sum((int(got.levels[0].rows[_pairs(F).index((int(c[0]), int(c[1])))]) + 31) // 32 for c in got.levels[1].cand)
    assert two == (len(got.levels[1].cand) > 256 or chunks > 1 << 17)
    assert waits == int(two)


def test_triples_of_large_features(ctx):
    """220 triples of features with 110,000 points: past 2^21 bitmap words."""
    wl = _places(_pairs(12), 10000)
    wl.thr, wl.max_size = 0.05, 3
    got, waits = _waits(ctx, wl)
    assert not got.levels[1].passed.any() and 3 * 220 * ((110000 + 31) // 32) > 1 << 21 and waits == 1


@pytest.mark.parametrize("groups,waits", [
    ([tuple(range(0, 7)), tuple(range(5, 12))], 0),            # 70 triples, all pass: one wait a level
    ([tuple(range(0, 13))], 1),                                 # 286 triples: two at level 3, one from then on
    ([tuple(range(0, 5))] + [p for p in _pairs(12) if p[1] > 4], 1),   # 10 of 220 triples pass: two at level 4
])
def test_levels_past_the_third(ctx, groups, waits):
    wl = _places(groups, 6)
    wl.thr = 0.05
    got, n = _waits(ctx, wl)
    assert len(got.levels) >= 3 and n == waits
