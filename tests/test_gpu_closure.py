"""DT closure at the shapes where its warps share work: starting sets around the
shares of a warp, rows around the 8 and 32 edges a lane takes, chains longer than
a run, buffers that fill, against a host search."""
import numpy as np
import pytest


pytestmark = pytest.mark.gpu


def rows(n, degree, seed):
    rng = np.random.default_rng(seed)
    u = np.repeat(np.arange(n), degree)
    v = (u + rng.integers(1, 4 * degree + 2, len(u))) % n
    return u, v


def path(n):
    return np.arange(n - 1), np.arange(1, n)


def tree(n, fan):
    v = np.arange(1, n)
    return (v - 1) // fan, v


CASES = {"one": lambda: (1, *path(1)), "path64": lambda: (65, *path(65)), "path": lambda: (5000, *path(5000)),
         "tree2": lambda: (40001, *tree(40001, 2)), "tree8": lambda: (40001, *tree(40001, 8)),
         "tree33": lambda: (40001, *tree(40001, 33)), "tree700": lambda: (40001, *tree(40001, 700))}
CASES.update({"rows%d" % d: lambda d=d: (6007, *rows(6007, d, d)) for d in (1, 7, 8, 9, 31, 32, 33)})


@pytest.mark.parametrize("starts", [1, 2, 31, 33, 609, 3000])
@pytest.mark.parametrize("case", sorted(CASES))
def test_closure(ctx, case, starts):
    import pagerank_gb300 as pg
    n, u, v = CASES[case]()
    rng = np.random.default_rng(starts)
    g = pg.Graph.from_edges(ctx, n, u.astype(np.uint32), v.astype(np.uint32), self_loops=True)
    xoff, xedg = g.download()[:2]
    src = rng.choice(n, min(starts, n), replace=False) if case[:4] == "rows" else np.arange(min(starts, n))
    src = np.sort(src).astype(np.uint32)
    seen = np.zeros(n, bool)
    for s in src:
        seen[xedg[xoff[s]:xoff[s + 1]]] = True   # the DF marking: out-neighbours of a batch's sources
    todo = list(np.flatnonzero(seen))
    while todo:
        x = todo.pop()
        for y in xedg[xoff[x]:xoff[x + 1]]:
            if not seen[y]:
                seen[y] = True
                todo.append(y)
    q = np.full(n, 1.0 / n)
    for expansion in (0, 1):   # 1: never by pull rounds
        _, res = pg.solve(ctx, g, pg.DYNAMIC_TRAVERSAL, None, (src, src), q,
                          pg.options(max_iterations=1, expansion=expansion))
        assert res["affected_initial"] == int(seen.sum())
    g.close()
