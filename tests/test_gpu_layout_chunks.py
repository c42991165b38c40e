"""LOW layouts of one, two and more source chunks, with and without hot sources,
on rows around the class bound (runs of LOW rows broken by longer ones): the
oracle's ranks bit for bit, from an uploaded graph and from an edge list."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hot", [-1, 500])
@pytest.mark.parametrize("chunks", [1, 2, 3, 8, 9])
def test_chunks(ctx, chunks, hot):
    import pagerank_gb300 as pg
    n, rng = 6007, np.random.default_rng(chunks)
    deg = rng.integers(0, 80, n)
    deg[::37] = 0
    deg[5:40] = np.arange(35) + 40
    v = np.repeat(np.arange(n), deg)
    u = rng.integers(0, n, len(v))
    key = np.unique(np.concatenate([u.astype(np.int64) * n + v, np.arange(n, dtype=np.int64) * (n + 1)]))
    off = np.zeros(n + 1, np.uint32)
    off[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    edg = (key % n).astype(np.uint32)
    xt = O.transpose(off, edg)
    want, it = O.solve("static", None, None, *xt)
    width = 0 if chunks == 1 else -(-n // chunks)
    width = (width + 31) // 32 * 32
    opts = pg.options(loop=pg.LOOP_GRAPH, chunk_vertices=width, hot_sources=hot)
    for g in (pg.Graph(ctx, *xt, off, edg),
              pg.Graph.from_edges(ctx, n, (key // n).astype(np.uint32), edg, self_loops=False)):
        r, res = pg.pagerank_static(ctx, g, opts)
        assert res["iterations"] == it and np.array_equal(r, want)
        g.close()
