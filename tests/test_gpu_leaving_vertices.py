"""Vertices that leave the affected set (DF-P): the copy of their ranks in the
other parity is refreshed by whichever warp takes their word, in the cooperative
loop (LOW rows by length and by word) and in the launched sweeps (by row, by
chunk)."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

GRAPHS = {"rmat": lambda pg: pg.graphs.rmat(15, 16, seed=11), "web": lambda pg: pg.graphs.weblike(60_001, seed=12)}


@pytest.mark.parametrize("prune", [1e-6, 1e-4, 1e-2])
@pytest.mark.parametrize("kind", sorted(GRAPHS))
def test_leaving_vertices(ctx, kind, prune):
    import pagerank_gb300 as pg
    xoff, xedg = GRAPHS[kind](pg)
    q, _ = O.solve("static", None, None, *O.transpose(xoff, xedg))
    for seed in (1, 2):
        batch = pg.graphs.random_batch(xoff, xedg, 60, 300, seed=seed)
        yoff, yedg = pg.graphs.apply_batch(xoff, xedg, *batch)
        yt = O.transpose(yoff, yedg)
        want, it = O.solve("prune_dynamic_frontier", yoff, yedg, *yt, *batch, q=q,
                           opts=O.options(prune_tolerance=prune))
        g = pg.Graph(ctx, *yt, yoff, yedg)
        for kw in ({}, {"loop": pg.LOOP_GRAPH}, {"loop": pg.LOOP_HOST, "chunk_vertices": 9000}):
            r, res = pg.solve(ctx, g, pg.PRUNE_DYNAMIC_FRONTIER, batch[:2], batch[2:], q,
                              pg.options(prune_tolerance=prune, **kw))
            assert res["iterations"] == it and np.array_equal(r, want), kw
        g.close()
