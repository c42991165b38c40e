"""Graphs whose out-degrees, as given, are not the lengths of the out-rows (accepted
without validation): contributions divide by the degrees, expansions follow the
rows, on every path alike."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("given", [1, 1024, 1500, 4000])
@pytest.mark.parametrize("length", [1024, 1025, 3000])
def test_expansion_follows_the_rows(ctx, length, given):
    import pagerank_gb300 as pg
    n = 5000
    rng = np.random.default_rng(length)
    u = np.concatenate([np.arange(n), np.zeros(length - 1, int), [1], rng.integers(2, n, 2 * n)])
    v = np.concatenate([np.arange(n), rng.choice(np.arange(2, n), length - 1, replace=False), [0],
                        rng.integers(2, n, 2 * n)])
    key = np.unique(u * n + v)
    xoff = np.zeros(n + 1, np.uint32)
    xoff[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    xedg = (key % n).astype(np.uint32)
    xtoff, xtedg, xtdat = O.transpose(xoff, xedg)
    assert xtdat[0] == length
    xtdat = xtdat.copy()
    xtdat[0] = given
    g = pg.Graph(ctx, xtoff, xtedg, xtdat, xoff, xedg)
    src, none = np.ones(1, np.uint32), np.zeros(0, np.uint32)   # vertex 1, whose only other neighbour is 0
    q = np.full(n, 1.0 / n)
    for mode in ("dynamic_frontier", "prune_dynamic_frontier"):
        want, it = O.solve(mode, xoff, xedg, xtoff, xtedg, xtdat, none, none, src, src, q=q)
        for kw in ({"expansion": 1}, {"expansion": 0}, {"loop": pg.LOOP_HOST}):
            r, res = pg.solve(ctx, g, pg.MODES[mode], None, (src, src), q, pg.options(**kw))
            assert res["iterations"] == it and np.array_equal(r, want), (mode, kw)
    g.close()
