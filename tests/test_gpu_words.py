"""LOW rows laid out by words: every mode's launched loop on graphs of long rows
(lengths 0 to 64 and longer in one word, a last word that is not full), before and
after a batch, against the oracle bit for bit; FP32-refined against the
cooperative loop, which reads the CSR."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu
DYN = ["naive_dynamic", "dynamic_traversal", "dynamic_frontier", "prune_dynamic_frontier"]


def graph(n, seed):
    rng = np.random.default_rng(seed)
    deg = rng.integers(0, 60, n)
    deg[: min(n, 66)] = np.arange(66)[: min(n, 66)]
    deg = np.minimum(deg, n - 1)
    v = np.repeat(np.arange(n), deg)
    key = np.unique(np.concatenate([rng.integers(0, n, len(v)) * n + v, np.arange(n) * (n + 1)]))
    off = np.zeros(n + 1, np.uint32)
    off[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    return off, (key % n).astype(np.uint32)


@pytest.mark.parametrize("hot", [-1, 0, 300])
@pytest.mark.parametrize("n", [64, 1000, 4099])
def test_words(ctx, n, hot):
    import pagerank_gb300 as pg
    xoff, xedg = graph(n, n)
    xt = O.transpose(xoff, xedg)
    g = pg.Graph(ctx, *xt, xoff, xedg)
    opts = lambda **kw: pg.options(loop=pg.LOOP_GRAPH, hot_sources=hot, **kw)
    q, it = O.solve("static", None, None, *xt)
    r, res = pg.pagerank_static(ctx, g, opts())
    assert res["iterations"] == it and np.array_equal(r, q)
    a, ra = pg.pagerank_static(ctx, g, opts(precision=pg.FP32_REFINE))
    b, rb = pg.pagerank_static(ctx, g, pg.options(precision=pg.FP32_REFINE))
    assert np.array_equal(a, b) and ra["iterations"] == rb["iterations"]
    batch = pg.graphs.random_batch(xoff, xedg, min(n // 3, 90), min(n, 40), seed=3)
    yoff, yedg = pg.graphs.apply_batch(xoff, xedg, *batch)
    yt = O.transpose(yoff, yedg)
    g.apply_batch(*batch)
    for mode in DYN:
        want, it = O.solve(mode, yoff, yedg, *yt, *batch, q=q)
        for int_adds in (-1, 1):
            r, res = pg.solve(ctx, g, pg.MODES[mode], batch[:2], batch[2:], q, opts(int_adds=int_adds))
            assert res["iterations"] == it and np.array_equal(r, want), (mode, int_adds)
    g.close()
