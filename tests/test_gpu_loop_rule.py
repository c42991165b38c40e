"""Which loop a large graph of mixed row lengths takes by itself: the cooperative one
where the order by length saves enough steps, launched sweeps where it does not, with
the same bits, iterations and weighted results either way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def draw(kind, n, per):
    rng = np.random.default_rng(8)
    if kind == "even":
        return rng.integers(0, n, n * per), rng.integers(0, n, n * per)
    # a fifth of the targets take most of the edges: rows of 1 beside rows of 20 and more
    v = np.where(rng.random(n * per) < 0.9, 8 * rng.integers(0, n // 8, n * per), rng.integers(0, n, n * per))
    return rng.integers(0, n, n * per), v


@pytest.mark.parametrize("kind, n, per, cooperative", [
    ("even", 1_500_000, 1, True), ("even", 1_600_000, 1, False), ("even", 1_600_001, 2, False),
    ("skewed", 1_600_000, 2, True),
])
def test_loop(ctx, kind, n, per, cooperative):
    import pagerank_gb300 as pg
    import torch
    from pagerank_gb300 import autograd as A
    u, v = (torch.from_numpy(x.astype(np.int32)).cuda() for x in draw(kind, n, per))
    g = pg.Graph.from_device_edges(ctx, n, u, v)
    q = np.random.default_rng(1).random(n) / n
    batch = np.arange(0, 300, dtype=np.uint32)
    for mode, dyn in ((pg.STATIC, False), (pg.NAIVE_DYNAMIC, False), (pg.DYNAMIC_TRAVERSAL, True),
                      (pg.DYNAMIC_FRONTIER, True), (pg.PRUNE_DYNAMIC_FRONTIER, True)):
        args = ((batch, batch), (batch[:0], batch[:0])) if dyn else (None, None)
        got = [pg.solve(ctx, g, mode, *args, None if mode == pg.STATIC else q, pg.options(loop=loop))
               for loop in (pg.LOOP_AUTO, pg.LOOP_GRAPH, pg.LOOP_HOST)]
        for r, res in got[1:]:
            assert res["iterations"] == got[0][1]["iterations"] and np.array_equal(r, got[0][0]), mode
        if not dyn:
            assert (got[0][1]["kernel_launches"] < got[1][1]["kernel_launches"]) == cooperative
    r32 = [pg.solve(ctx, g, pg.STATIC, opts=pg.options(precision=pg.FP32_REFINE, loop=loop))[0]
           for loop in (pg.LOOP_AUTO, pg.LOOP_GRAPH)]
    assert np.array_equal(*r32)
    A.set_weights(ctx, g, torch.rand(g.size()[1], device="cuda") + 0.5)
    w = [A.solve_weighted(ctx, g, opts=pg.options(loop=loop))[0] for loop in (pg.LOOP_AUTO, pg.LOOP_HOST)]
    assert float((w[0] - w[1]).abs().max()) <= 1e-12 * float(w[1].max())
    g.close()
