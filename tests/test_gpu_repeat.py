"""Repeated timed solves (options.repeat): every repetition starts from the caller's
ranks, so the result is that of one solve."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu
MODES = ["static", "naive_dynamic", "dynamic_traversal", "dynamic_frontier", "prune_dynamic_frontier"]


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("kw", [{}, {"loop": 2}, {"precision": 1}], ids=["auto", "graph", "refine"])
def test_repetitions_start_alike(ctx, mode, kw):
    import pagerank_gb300 as pg
    xoff, xedg = pg.graphs.rmat(11, 16, seed=5)
    q, _ = O.solve("static", None, None, *O.transpose(xoff, xedg))
    batch = pg.graphs.random_batch(xoff, xedg, 20, 80, seed=2)
    yoff, yedg = pg.graphs.apply_batch(xoff, xedg, *batch)
    g = pg.Graph(ctx, *O.transpose(yoff, yedg), yoff, yedg)
    got = [pg.solve(ctx, g, pg.MODES[mode], batch[:2], batch[2:], q, pg.options(repeat=k, **kw)) for k in (1, 3)]
    assert got[0][1]["iterations"] == got[1][1]["iterations"]
    assert np.array_equal(got[0][0], got[1][0])
    g.close()
