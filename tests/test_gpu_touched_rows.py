"""Batches on rows of every length around the steps of the merge (32, 64, 512 ids a
row) and of the carried layouts (8 lanes a row, 64 ids): the graph against the host's,
Static by the carried layouts, plain and with chunks, against the oracle."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu
LENGTHS = {"short": list(range(1, 67)) * 3, "long": [31, 32, 33, 63, 64, 65, 66, 127, 128, 129, 255, 256, 257,
                                                     511, 512, 513, 514, 600, 769, 1025]}


@pytest.mark.parametrize("chunk", [0, 400])
@pytest.mark.parametrize("rows", sorted(LENGTHS))
def test_apply(ctx, rows, chunk):
    import pagerank_gb300 as pg
    n, rng = 1500, np.random.default_rng(6)
    key = {(int(v), int(v)) for v in range(n)}
    for u, d in enumerate(LENGTHS[rows]):   # out-rows, and in-rows of the same lengths further up
        key |= {(u, int(v)) for v in rng.choice(n, d, replace=False)}
        key |= {(int(v), 700 + u) for v in rng.choice(n, d, replace=False)}
    key = np.array(sorted(key))
    off = np.zeros(n + 1, np.uint32)
    off[1:] = np.cumsum(np.bincount(key[:, 0], minlength=n))
    edg = key[:, 1].astype(np.uint32)
    g = pg.Graph(ctx, *O.transpose(off, edg), off, edg)
    opts = pg.options(loop=pg.LOOP_GRAPH, chunk_vertices=chunk, hot_sources=64)
    for step in range(4):
        pg.solve(ctx, g, pg.STATIC, opts=opts)   # a layout to carry
        loops = key[:, 0] == key[:, 1]
        gone = key[~loops][rng.choice((~loops).sum(), [1, 60, 700, 2000][step], replace=False)]
        have = {tuple(x) for x in key}
        new = {(int(a), int(b)) for a, b in zip(rng.integers(0, 300, 900), rng.integers(0, n, 900))}
        new |= {(int(b), 700 + int(a)) for a, b in zip(rng.integers(0, 220, 900), rng.integers(0, n, 900))}
        new = np.array(sorted(new - have))
        gone = np.array(sorted(map(tuple, gone)))
        left = np.array(sorted((have - {tuple(x) for x in gone}) | {tuple(x) for x in new}))
        cols = [np.ascontiguousarray(x.astype(np.uint32)) for x in (gone[:, 0], gone[:, 1], new[:, 0], new[:, 1])]
        g.apply_batch(*cols)
        key = left
        off[1:] = np.cumsum(np.bincount(key[:, 0], minlength=n))
        edg = key[:, 1].astype(np.uint32)
        xt = O.transpose(off, edg)
        for a, b in zip(g.download(), (off, edg, *xt)):
            assert np.array_equal(a, b), step
        want, it = O.solve("static", None, None, *xt)
        r, res = pg.solve(ctx, g, pg.STATIC, opts=opts)
        assert res["iterations"] == it and np.array_equal(r, want), step
    g.close()
