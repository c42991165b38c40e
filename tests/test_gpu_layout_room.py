"""A batch whose deletions bring rows down to the LOW class: the carried layout
has room for all of their remaining edges."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("down,up", [(1, 0), (700, 0), (700, 3), (3, 700)])
def test_rows_crossing_the_low_bound(ctx, down, up):
    import pagerank_gb300 as pg
    n, rng = 30011, np.random.default_rng(down + up)
    rows = rng.choice(n, down + up, replace=False)
    u, v = [np.arange(n)], [np.arange(n)]
    for i, x in enumerate(rows):  # in-degree 65 before a deletion, 64 before an insertion
        src = rng.choice(np.delete(np.arange(n), x), 64 if i < down else 63, replace=False)
        u.append(src)
        v.append(np.full(len(src), x))
    u, v = np.concatenate(u).astype(np.uint32), np.concatenate(v).astype(np.uint32)
    key = np.unique(u.astype(np.int64) * n + v)
    g = pg.Graph.from_edges(ctx, n, (key // n).astype(np.uint32), (key % n).astype(np.uint32), self_loops=False)
    opts = pg.options(loop=pg.LOOP_GRAPH, hot_sources=64)
    pg.pagerank_static(ctx, g, opts)   # builds the layout
    drop = np.array([next(k for k in key[key % n == x] if k // n != x) for x in rows[:down]], np.int64)
    have = set(key.tolist())
    add = np.array([next(s * n + x for s in range(n) if s * n + x not in have) for x in rows[down:]], np.int64)
    drop, add = np.unique(drop), np.unique(add)
    part = lambda k: ((k // n).astype(np.uint32), (k % n).astype(np.uint32))
    g.apply_batch(*part(drop), *part(add))
    keep = [pg.Graph.from_edges(ctx, n, u, v) for _ in range(3)]   # what follows the layout in memory
    r, res = pg.pagerank_static(ctx, g, opts)
    now = np.union1d(np.setdiff1d(key, drop), add)
    off = np.zeros(n + 1, np.uint32)
    off[1:] = np.cumsum(np.bincount(now // n, minlength=n))
    want, it = O.solve("static", None, None, *O.transpose(off, (now % n).astype(np.uint32)))
    assert res["iterations"] == it and np.array_equal(r, want)
    for x in keep + [g]:
        x.close()
