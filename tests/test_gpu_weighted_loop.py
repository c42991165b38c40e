"""The weighted solve and the adjoint as one cooperative kernel (the default of
small and medium graphs) against the launched sweeps, where rows meet their
class bounds, and weights set again on a graph that keeps its positions."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pg():
    import pagerank_gb300
    return pagerank_gb300


def _bounds(pg):
    """Out- and in-degrees around 64, 1024 and 4096 (n = 4200)."""
    rng = np.random.default_rng(1)
    n = 4200
    u, v = [np.arange(n)], [np.arange(n)]
    for at, d in enumerate([2, 33, 63, 64, 65, 96, 128, 1023, 1024, 1025, 2048, 4095, 4096, 4097, 4100]):
        other = rng.choice(np.delete(np.arange(n), at), d - 1, replace=False)
        u += [np.full(d - 1, at), other]
        v += [other, np.full(d - 1, (at + 20))]
    key = np.unique(np.concatenate(u).astype(np.int64) * n + np.concatenate(v))
    off = np.zeros(n + 1, np.uint32)
    off[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    return off, (key % n).astype(np.uint32)


CASES = {"one": lambda pg: pg.graphs.grid(1), "bounds": _bounds, "rmat": lambda pg: pg.graphs.rmat(12, 16, seed=3),
         "web": lambda pg: pg.graphs.weblike(3001, dmax=900, window=512, seed=9)}


@pytest.mark.parametrize("case", sorted(CASES))
def test_loop_equals_launched_sweeps(pg, ctx, case):
    import torch
    from pagerank_gb300 import autograd as A
    xoff, xedg = CASES[case](pg)
    n, m = len(xoff) - 1, len(xedg)
    g = pg.Graph(ctx, *O.transpose(xoff, xedg), xoff, xedg)
    gen = torch.Generator(device="cuda").manual_seed(5)
    w1, w2 = (0.5 + torch.rand(m, generator=gen, device="cuda") for _ in range(2))
    t = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)
    goal = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) - 0.5
    got = {}
    for loop in (pg.LOOP_AUTO, pg.LOOP_HOST, pg.LOOP_AUTO):
        o = pg.options(tolerance=1e-14, max_iterations=500, loop=loop)
        A.set_weights(ctx, g, w2)
        A.set_weights(ctx, g, w1)
        r, res = A.solve_weighted(ctx, g, t, opts=o)
        d = A.adjoint(ctx, g, r, goal, t, o, want_lambda=True)
        key = "again" if loop in got else loop
        got[key] = [r, d["lambda"], d["grad_w"], d["grad_t"], torch.tensor(d["grad_alpha"])]
    for a, b, c in zip(got[pg.LOOP_AUTO], got[pg.LOOP_HOST], got["again"]):
        scale = float(b.abs().max()) + 1e-300
        assert float((a - b).abs().max()) <= 1e-12 * scale   # rows of 1025 to 4096 edges are summed in another order
        assert torch.equal(a, c)
    # the rows of P sum to one: ranks keep the teleport vector's mass
    r = got[pg.LOOP_AUTO][0]
    assert abs(float(r.sum()) / float(t.sum()) - 1) < 1e-10
    for cap in (0, 1, 2, 3):
        both = [A.solve_weighted(ctx, g, t, opts=pg.options(max_iterations=cap, tolerance=0.0, loop=loop))
                for loop in (pg.LOOP_AUTO, pg.LOOP_HOST)]
        assert both[0][1]["iterations"] == both[1][1]["iterations"] == cap
        assert float((both[0][0] - both[1][0]).abs().max()) <= 1e-12 * float(t.max())
    g.close()


def test_plan_stays_after_autotune(pg, ctx):
    import torch
    from pagerank_gb300 import autograd as A
    g = pg.Graph.from_out_csr(ctx, *pg.graphs.rmat(12, 16, seed=3))
    n, m = g.size()
    A.set_weights(ctx, g, 0.5 + torch.rand(m, generator=torch.Generator(device="cuda").manual_seed(5), device="cuda"))
    goal = torch.ones(n, dtype=torch.float64, device="cuda")
    r, _ = A.solve_weighted(ctx, g)
    before = A.adjoint(ctx, g, r, goal)
    pg.autotune(ctx, g)
    after = A.adjoint(ctx, g, r, goal)
    assert torch.equal(before["grad_w"], after["grad_w"])
    # one kernel for the loop, not three a sweep
    assert after["result"]["kernel_launches"] < before["result"]["kernel_launches"] + after["result"]["iterations"]
    g.close()
