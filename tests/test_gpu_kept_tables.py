"""Kept tables are turned into rows on the device and copied behind each level's fill: tables of zero rows, of one,
of many, several levels in one mine and several jobs in one batch, tables in host memory, and more than the
staging's 64 MiB (copied in parts), against the oracle's tables row for row."""
import numpy as np
import pytest

import colo
from colo import gen
from colo.gen import Workload
from helpers import assert_same_trace, oracle_for

pytestmark = pytest.mark.gpu


def _blob(per, features, seed):
    rng = np.random.default_rng(seed)
    n = per * features
    x, y = (rng.normal(50, 0.4, n).astype(np.float32) for _ in range(2))
    return Workload("blob", x, y, np.repeat(np.arange(features, dtype=np.int32), per),
                    np.array([0, 0, 100, 100], np.float32), 12.0, 0.1, [], 3)


@pytest.mark.parametrize("host", [False, True])
def test_many_levels_and_jobs(host):
    ctx = colo.Context(0)
    jobs = [gen.config(0), gen.config(1, scale=0.03), _blob(9, 5, 1), gen.config(0, seed=5)]
    dss = [colo.Dataset.from_arrays(ctx, w.x, w.y, w.fid, w.bounds) for w in jobs]
    refs = [oracle_for(ctx, w, keep_tables=True) for w in jobs]
    for mode in (colo.MODE_BATCHED, colo.MODE_PLAIN):
        ps = [colo.default_params(w.R, w.thr, mode, max_size=w.max_size, keep_tables=True, host_tables=host) for w in jobs]
        first = 0   # a batched job's tables number the points of the whole batch
        for w, got, ref in zip(jobs, ctx.mine_batch(dss, ps), refs):
            for lev in got.levels:
                lev.tables = {c: t - np.uint32(first) for c, t in lev.tables.items()}
            assert_same_trace(got, ref, tables=True)
            first += w.n if mode == colo.MODE_BATCHED else 0


def test_more_than_the_staging():
    """Two features of 3,100 points and one of a single point, all within one reach: a pair table of 9.6 million rows
    (77 MB), checked without the oracle: every point of one feature with every point of the other, rows in order of
    the first."""
    wl = _blob(3100, 3, 2)
    keep = 2 * 3100 + 1
    wl.x, wl.y, wl.fid = wl.x[:keep], wl.y[:keep], wl.fid[:keep]
    ctx = colo.Context(0)
    ds = colo.Dataset.from_arrays(ctx, wl.x, wl.y, wl.fid, wl.bounds)
    got = ctx.mine(ds, colo.default_params(wl.R, wl.thr, max_size=3, keep_tables=True))
    lev = got.levels[0]
    assert len(lev.tables) == 1   # {0, 1}, the prefix of {0, 1, 2}
    a, b = np.divmod(np.arange(3100 * 3100, dtype=np.int64), 3100)
    for c, t in lev.tables.items():
        f, g = lev.cand[c]
        assert np.array_equal(t[:, 0], a + 3100 * int(f)) and np.array_equal(np.sort(t[:, 1].reshape(3100, 3100), axis=1).ravel(), b + 3100 * int(g))
