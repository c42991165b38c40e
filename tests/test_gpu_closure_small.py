"""DT closure of small graphs, whose switch to pull rounds (a sixteenth of the
vertices) lies among the first few marked ones: fewer, as many and more of them
than that, and no more than eight times those done."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("marked", range(1, 9))
@pytest.mark.parametrize("n", [15, 16, 17, 33, 64, 100, 111, 112, 128])
def test_small_closure(ctx, n, marked):
    import pagerank_gb300 as pg
    # vertex 0 has `marked` out-neighbours with its loop, the others a path and a few chords
    u = np.concatenate([np.arange(n), np.zeros(marked - 1, int), np.arange(1, n - 1), np.arange(1, n, 5)])
    v = np.concatenate([np.arange(n), n - 1 - np.arange(marked - 1), np.arange(2, n), (3 * np.arange(1, n, 5)) % n])
    key = np.unique(u * n + v)
    xoff = np.zeros(n + 1, np.uint32)
    xoff[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    xedg = (key % n).astype(np.uint32)
    assert xoff[1] == marked
    xt = O.transpose(xoff, xedg)
    src, none = np.zeros(1, np.uint32), np.zeros(0, np.uint32)
    q = np.full(n, 1.0 / n)
    want, it = O.solve("dynamic_traversal", xoff, xedg, *xt, none, none, src, src, q=q)
    seen = np.zeros(n, bool)
    todo = list(xedg[:marked])
    while todo:
        x = todo.pop()
        if not seen[x]:
            seen[x] = True
            todo.extend(xedg[xoff[x]:xoff[x + 1]])
    g = pg.Graph(ctx, *xt, xoff, xedg, validate=True)
    for expansion in (0, 1, 2):
        r, res = pg.solve(ctx, g, pg.DYNAMIC_TRAVERSAL, None, (src, src), q, pg.options(expansion=expansion))
        assert res["affected_initial"] == int(seen.sum()), expansion
        assert res["iterations"] == it and np.array_equal(r, want), expansion
    g.close()
