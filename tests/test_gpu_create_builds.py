"""A graph created from host CSRs builds what its default solves read and nothing
else, and every solve builds what it still misses."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["rmat", "web", "grid"])
def test_host_graph_holds_no_unused_layout(ctx, kind):
    import pagerank_gb300 as pg
    xoff, xedg = {"rmat": lambda: pg.graphs.rmat(17, 16, seed=3), "web": lambda: pg.graphs.weblike(60_001, seed=4),
                  "grid": lambda: pg.graphs.grid(700, seed=5)}[kind]()
    n = len(xoff) - 1
    used = lambda: pg.graph_pool_stats()["used"]
    at = used()
    g = pg.Graph.from_edges(ctx, n, np.repeat(np.arange(n), np.diff(xoff.astype(np.int64))), xedg, self_loops=False)
    from_edges = used() - at
    g.close()
    at = used()
    xt = O.transpose(xoff, xedg)
    g = pg.Graph(ctx, *xt, xoff, xedg)
    in_degree = np.diff(xt[0].astype(np.int64))
    layout = 4 * int(in_degree[in_degree <= 64].sum())
    assert layout > 1 << 20 and used() - at < from_edges + layout // 4
    # every way to solve it, the first solve of a graph
    want, it = O.solve("static", None, None, *xt)
    for kw in ({}, {"loop": pg.LOOP_GRAPH}, {"loop": pg.LOOP_HOST, "hot_sources": 500}, {"chunk_vertices": 20000}):
        x = pg.Graph(ctx, *xt, xoff, xedg)
        r, res = pg.pagerank_static(ctx, x, pg.options(**kw))
        assert res["iterations"] == it and np.array_equal(r, want), kw
        x.close()
    g.close()
