"""The one-pass neighbourhood lists and the join at the edges of their paths: cells whose anchors are listed by
one thread (up to 32) or by the whole warp, lists merged by one thread (up to 128 runs and 512 points) or by the
warp, runs of up to 32 points and longer ones, anchors of up to 64 targets and longer ones, every number of lanes
per anchor, and more targets than the first allocation holds (four a point plus 65,536), which builds the lists
again.  The neighbour lists equal the oracle's exactly."""
import numpy as np
import pytest

import colo
import oracle
from helpers import resolve_ambiguous

pytestmark = pytest.mark.gpu


def _check(x, y, fid, bounds, R, widths=(0,)):
    ctx = colo.Context(0)
    ds = colo.Dataset.from_arrays(ctx, x, y, fid, bounds)
    res = resolve_ambiguous(ctx, x, y, fid, R)
    o_offs, o_nbr, unres = oracle.neighbors(x, y, fid, bounds, R, res=res)
    assert unres == 0
    for width in widths:
        ctx.set_join_group(width)
        offs, nbr = ctx.stage_neighbors(ds, R)
        assert np.array_equal(offs, o_offs)
        assert np.array_equal(nbr, o_nbr)
        assert nbr.size > 0


@pytest.mark.parametrize("per", [1, 15, 16, 17, 40])
@pytest.mark.parametrize("cells", [1, 31, 33])
def test_anchors_per_cell(per, cells):
    """`cells` separate cells with `per` points of each of three features: 2 * per anchors a cell."""
    rng = np.random.default_rng(per * 100 + cells)
    x = np.concatenate([np.concatenate([30.0 * c + rng.uniform(0.0, 10.0, per) for c in range(cells)])
                        for _ in range(3)]).astype(np.float32)
    y = rng.uniform(0.0, 10.0, len(x)).astype(np.float32)
    fid = np.repeat(np.arange(3, dtype=np.int32), per * cells)
    _check(x, y, fid, np.array([0.0, 0.0, 30.0 * cells + 20.0, 40.0], np.float32), 10.0)


@pytest.mark.parametrize("features,side", [(40, 45), (15, 20), (16, 20), (3, 330)])
def test_list_lengths(features, side):
    """Every cell of a side x side grid holds one point of every feature: nine times (features - 1) targets an
    inner cell (126 and 135 runs: both sides of the long-list limit).  40 features on 45 x 45 cells need more than
    four targets a point; 330 x 330 cells are more than the grid's warps take one each."""
    rng = np.random.default_rng(features)
    gx, gy = np.meshgrid(np.arange(side), np.arange(side))
    x = np.concatenate([(gx.ravel() + rng.uniform(0.01, 0.99, side * side)) * 10.0 for _ in range(features)])
    y = np.concatenate([(gy.ravel() + rng.uniform(0.01, 0.99, side * side)) * 10.0 for _ in range(features)])
    fid = np.repeat(np.arange(features, dtype=np.int32), side * side)
    _check(x.astype(np.float32), y.astype(np.float32), fid, np.array([0, 0, 10 * side, 10 * side], np.float32), 10.0)


@pytest.mark.parametrize("per", [31, 32, 33, 63, 64, 65, 127, 128, 129, 256, 513, 700])
def test_long_runs(per):
    """Two features with `per` points in a cell and one point in a far one: runs of `per` points, `per` targets an
    anchor (both sides of 32 a run, 64 an anchor and 512 a list), and a single-target anchor beside them."""
    rng = np.random.default_rng(per)
    x = np.concatenate([rng.uniform(20, 30, per), [75.0], rng.uniform(20, 30, per), [76.0], [25.0]]).astype(np.float32)
    y = np.concatenate([rng.uniform(20, 30, per), [75.0], rng.uniform(20, 30, per), [76.0], [25.0]]).astype(np.float32)
    fid = np.concatenate([np.zeros(per + 1), np.ones(per + 1), [2]]).astype(np.int32)
    _check(x, y, fid, np.array([0, 0, 100, 100], np.float32), 10.0, widths=(0,) + colo.JOIN_WIDTHS)
