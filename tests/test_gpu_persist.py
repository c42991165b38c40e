"""The iteration loop as one cooperative kernel (the default of graphs up to
some tens of millions of edges): the ranks, iteration counts and edge counts
of the launched loops bit for bit, and the oracle's, where rows, words and
expansions meet their edges."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu
DYN = ["naive_dynamic", "dynamic_traversal", "dynamic_frontier", "prune_dynamic_frontier"]


@pytest.fixture(scope="module")
def pg():
    import pagerank_gb300
    pagerank_gb300.load()
    return pagerank_gb300


def _rows(n, lengths, seed):
    """Out-CSR with a loop on every vertex and rows of the given in-degrees."""
    rng = np.random.default_rng(seed)
    u = [np.arange(n)]
    v = [np.arange(n)]
    for at, d in enumerate(lengths):
        src = rng.choice(np.delete(np.arange(n), at), d - 1, replace=False)
        u.append(src)
        v.append(np.full(d - 1, at))
    key = np.unique(np.concatenate(u).astype(np.int64) * n + np.concatenate(v))
    off = np.zeros(n + 1, np.uint32)
    off[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    return off, (key % n).astype(np.uint32)


CASES = {
    "one": lambda pg: _rows(1, [], 0),
    "33": lambda pg: _rows(33, [5, 32, 33], 1),
    # around the class bounds (64 | 65, 4096 | 4097), multiples of 32 and 256, and HIGH remainders
    "bounds": lambda pg: _rows(8192 + 31, [2, 3, 4, 5, 8, 63, 64, 65, 96, 97, 128, 129, 255, 256, 257, 288, 511, 512,
                                           513, 2049, 4095, 4096, 4097, 4353, 6145, 8000], 2),
    "rmat": lambda pg: pg.graphs.rmat(13, 16, seed=3),
    "hubs": lambda pg: pg.graphs.weblike(20_001, alpha=1.6, dmin=3.0, dmax=15000, seed=4),  # out-degrees over 1024
    "grid": lambda pg: pg.graphs.grid(57, seed=5),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_equals_oracle_and_launched_loop(pg, ctx, case):
    xoff, xedg = CASES[case](pg)
    n = len(xoff) - 1
    xt = O.transpose(xoff, xedg)
    q, it = O.solve("static", None, None, *xt)
    g = pg.Graph(ctx, *xt, xoff, xedg)
    r, res = pg.pagerank_static(ctx, g)
    assert res["iterations"] == it and np.array_equal(r, q)
    batch = pg.graphs.random_batch(xoff, xedg, min(n // 3, 40), min(n, 200), seed=9)
    yoff, yedg = pg.graphs.apply_batch(xoff, xedg, *batch)
    yt = O.transpose(yoff, yedg)
    y = pg.Graph(ctx, *yt, yoff, yedg)
    for mode in DYN:
        want, it = O.solve(mode, yoff, yedg, *yt, *batch, q=q)
        for expansion in (0, 1, 2):
            r, a = pg.solve(ctx, y, pg.MODES[mode], batch[:2], batch[2:], q, pg.options(expansion=expansion))
            assert a["iterations"] == it and np.array_equal(r, want), (mode, expansion)
        r, b = pg.solve(ctx, y, pg.MODES[mode], batch[:2], batch[2:], q, pg.options(loop=pg.LOOP_GRAPH))
        assert np.array_equal(r, want)
        for key in ("iterations", "edges_processed", "affected_initial", "last_delta"):
            assert a[key] == b[key], (mode, key)
        for cap in (0, 1, 2, 3):
            want, it = O.solve(mode, yoff, yedg, *yt, *batch, q=q, opts=O.options(max_iterations=cap))
            r, a = pg.solve(ctx, y, pg.MODES[mode], batch[:2], batch[2:], q, pg.options(max_iterations=cap))
            assert a["iterations"] == it and np.array_equal(r, want), (mode, cap)
    g.close()
    y.close()
