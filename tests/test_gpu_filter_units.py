"""The level filter's units: every number of candidates per unit, drivers with one candidate, as many as a unit and
more, driver lists on both sides of 32 cells, counters in shared memory and (many candidates) in global memory, and
mask widths on both sides of the one that loads or shuffles a candidate's mask.  Bounds equal a brute-force count."""
import numpy as np
import pytest

import colo

pytestmark = pytest.mark.gpu


def _bounds(x, y, fid, R, gx, gy, cand):
    F = int(fid.max()) + 1
    cells = np.zeros((F, gy, gx), np.int64)
    np.add.at(cells, (fid, (y / R).astype(int), (x / R).astype(int)), 1)
    has = cells > 0
    quad = has[:, :-1, :-1] | has[:, :-1, 1:] | has[:, 1:, :-1] | has[:, 1:, 1:]
    out = np.zeros(cand.shape, np.int64)
    for i, c in enumerate(cand):
        full = np.logical_and.reduce(quad[c])
        u = np.zeros((gy, gx), bool)
        u[:-1, :-1] |= full
        u[:-1, 1:] |= full
        u[1:, :-1] |= full
        u[1:, 1:] |= full
        out[i] = [cells[f][u].sum() for f in c]
    return out


@pytest.mark.parametrize("features", [8, 40, 100, 130, 224])
@pytest.mark.parametrize("unit", [8, 16, 32])
def test_bounds_match_brute_force(features, unit):
    rng = np.random.default_rng(features)
    R, side = np.float32(10.0), 12
    n = features * 40
    fid = np.sort(rng.integers(0, features, n)).astype(np.int32)
    fid[:features] = np.arange(features)
    fid = np.sort(fid)
    x, y = (rng.uniform(0, 120, n).astype(np.float32) for _ in range(2))
    first = np.array([[0, b, c] for b in range(1, min(features, 12)) for c in range(b + 1, min(features, 12))], np.uint32)
    many = np.sort(np.array([rng.choice(features, 3, replace=False) for _ in range(4000)]), axis=1).astype(np.uint32)
    ctx = colo.Context(0)
    ctx.set_tuning(filter_unit=unit)
    ds = colo.Dataset.from_arrays(ctx, x, y, fid, np.array([0, 0, 120, 110], np.float32))
    for cand in (first, many):   # 4000 candidates: 20,000 counters, more than fit in shared memory
        ub, _ = ctx.stage_filter(ds, float(R), 0.1, cand)
        assert np.array_equal(ub.astype(np.int64), _bounds(x, y, fid, R, side, side, cand))
