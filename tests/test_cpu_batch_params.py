"""mine_batch reads its parameters once, in order: any iterable that it took stays accepted (a generator, fewer than the
datasets), and what a result looks for follows the parameters that the mine was given.  The library's call is a
stand-in; no GPU."""
from types import SimpleNamespace

import pytest

import colo


class _Lib:
    """Stands in for the library: records the parameters of the call and hands out null results."""

    def colo_mine_batch(self, ctx, datasets, params, n, outs):
        self.seen = [(float(params[i].distance), int(params[i].keep_tables), int(params[i].reserved[0])) for i in range(n)]
        return colo.OK


def _context():
    ctx = colo.Context.__new__(colo.Context)
    ctx.lib, ctx.h = _Lib(), None
    return ctx


@pytest.mark.parametrize("given", [list, tuple, iter, lambda ps: (p for p in ps)])
def test_any_iterable_of_parameters(given):
    ps = [colo.default_params(1.0 + i, 0.5, keep_tables=i == 1) for i in range(3)]
    ps[2].reserved[0] |= 2
    ctx = _context()
    got = ctx.mine_batch([SimpleNamespace(h=None)] * 3, given(ps))
    assert ctx.lib.seen == [(1.0, 0, 0), (2.0, 1, 0), (3.0, 0, 2)]
    assert [r._has_tables for r in got] == [False, True, False]
    assert [r._has_features for r in got] == [False, False, True]


def test_fewer_parameters_than_datasets():
    ctx = _context()
    got = ctx.mine_batch([SimpleNamespace(h=None)] * 2, [colo.default_params(4.0, 0.5, keep_tables=True)])
    assert ctx.lib.seen == [(4.0, 1, 0), (0.0, 0, 0)] and len(got) == 2
