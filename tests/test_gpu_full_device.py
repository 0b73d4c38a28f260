"""Mines on a device that is nearly full (colo_params.reserved[3] limits what a mine's buffers may take; allocations past
it are refused as on a full device): what fits when sizes are read back before the arrays over cells are laid out is
mined, and with its tables on the device, though the arrays laid out by bounds are larger.  With less, tables go to host
memory, and below that the mine is refused; every mine that is not refused has the result of an empty device."""
import numpy as np
import pytest

import colo
from helpers import FIELDS
from test_gpu_layouts import _points

pytestmark = pytest.mark.gpu

ERR_NOMEM = 6
EXACT = -1   # reserved[2]: sizes are counted before arrays are laid out


@pytest.fixture(scope="module")
def ctx():
    c = colo.Context(0)
    yield c
    c.set_model(None)


def _mine(ctx, dss, wl, mode, budget=0, kib=0, keep=False):
    ps = []
    for _ in dss:
        p = colo.default_params(wl.R, wl.thr, mode, max_size=wl.max_size, keep_tables=keep, profile=True)
        p.reserved[2], p.reserved[3] = kib, budget
        ps.append(p)
    return ctx.mine_batch(dss, ps)


def _fits(ctx, dss, wl, mode, budget, kib):
    try:
        return _mine(ctx, dss, wl, mode, budget, kib)[0].counters["host_table_bytes"] == 0
    except colo.ColoError as e:
        assert e.status == ERR_NOMEM
        return False


def _least(ctx, dss, wl, mode, kib):
    """The least budget (KiB, to 8) with which a layout mines with its tables on the device."""
    lo, hi = 64, 1 << 20
    assert _fits(ctx, dss, wl, mode, hi, kib) and not _fits(ctx, dss, wl, mode, lo, kib)
    while hi - lo > 8:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if _fits(ctx, dss, wl, mode, mid, kib) else (mid, hi)
    return hi


def _same(a, b, tables=False):
    assert len(a.levels) == len(b.levels) >= 2
    for p, q in zip(a.levels, b.levels):
        for f in FIELDS + ("pi",):
            assert np.array_equal(getattr(p, f), getattr(q, f)), (p.k, f)
        if tables:
            assert set(p.tables) == set(q.tables) and all(np.array_equal(t, q.tables[c]) for c, t in p.tables.items())


# lines: few and short tables (the arrays are what counts), and tables of several times the arrays
@pytest.mark.parametrize("lines", [20, 7])
@pytest.mark.parametrize("mode", [colo.MODE_BATCHED, colo.MODE_PLAIN, colo.MODE_LEARNED])
@pytest.mark.parametrize("jobs", [1, 3])
def test_what_fits_with_sizes_read_back(ctx, lines, mode, jobs):
    wl = _points(20000, 6, 6000.0, lines, 7)
    wl.max_size = 4
    ctx.set_model(colo.load_model() if mode == colo.MODE_LEARNED else None)
    dss = [colo.Dataset.from_arrays(ctx, wl.x, wl.y, wl.fid, wl.bounds) for _ in range(jobs)]
    for ds in dss:
        ds.upload()
    whole = _mine(ctx, dss, wl, mode)
    assert "host cell_masks" not in whole[0].kernels
    budget = _least(ctx, dss, wl, mode, EXACT)
    got = _mine(ctx, dss, wl, mode, budget)
    assert got[0].counters["host_table_bytes"] == 0
    for a, b in zip(whole, got):
        _same(a, b)
    assert "host cell_masks" in got[0].kernels or "host cell_heads" in got[0].kernels   # not by bounds


@pytest.mark.parametrize("mode", [colo.MODE_BATCHED, colo.MODE_PLAIN])
def test_any_budget(ctx, mode):
    """From too little for anything to enough for everything, tables kept."""
    wl = _points(20000, 6, 6000.0, 7, 7)
    wl.max_size = 4
    ds = colo.Dataset.from_arrays(ctx, wl.x, wl.y, wl.fid, wl.bounds)
    ds.upload()
    whole, = _mine(ctx, [ds], wl, mode, keep=True)
    refused = on_host = on_device = 0
    for budget in [256, 512, 1024] + list(range(1536, 8192, 128)) + list(range(8192, 1 << 16, 4096)):
        try:
            got, = _mine(ctx, [ds], wl, mode, budget, keep=True)
        except colo.ColoError as e:
            assert e.status == ERR_NOMEM and not on_host and not on_device, budget
            refused += 1
            continue
        _same(whole, got, tables=True)
        on_host += got.counters["host_table_bytes"] > 0
        on_device += got.counters["host_table_bytes"] == 0
    assert refused >= 3 and on_host >= 3 and on_device >= 1
