"""Tuning caches written for the join that gave each anchor a group of lanes (join=<lanes>) are not applied to the one
that tiles anchors: such a line is skipped and the shape is timed.  Tuning a dataset without points sets the default
width."""
import re

import numpy as np
import pytest

import colo
from colo import gen

pytestmark = pytest.mark.gpu


def test_lines_of_the_grouped_join_are_skipped(tmp_path):
    cache = tmp_path / "tuning.txt"
    wl = gen.config(0)
    ctx = colo.Context(0)
    ds = colo.Dataset.from_arrays(ctx, wl.x, wl.y, wl.fid, wl.bounds)
    prm = colo.default_params(wl.R, wl.thr, colo.MODE_BATCHED, max_size=wl.max_size)
    assert not ctx.autotune_all(ds, prm, cache=str(cache))["from_cache"]
    line = cache.read_text()
    old = re.sub(r" \w+=\d+ funit=", " join=8 funit=", line)
    assert old.startswith("colo-tune 2 n=") and old.count("join=8") == 1
    cache.write_text(old)
    again = ctx.autotune_all(ds, prm, cache=str(cache))
    assert not again["from_cache"]
    assert cache.read_text().startswith(old) and len(cache.read_text().splitlines()) == 2
    assert ctx.autotune_all(ds, prm, cache=str(cache))["from_cache"]


def test_no_points_tune_to_the_default():
    ctx = colo.Context(0)
    none = np.zeros(0, np.float32)
    ds = colo.Dataset.from_arrays(ctx, none, none, np.zeros(0, np.int32), np.array([0, 0, 1, 1], np.float32))
    assert ctx.autotune(ds, colo.default_params(1.0, 0.5))["join_group"] == 1
