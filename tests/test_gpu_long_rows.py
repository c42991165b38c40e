"""Graphs whose long rows decide how the cooperative loops share them out: many rows
of 1025 to 4096 (by warp), a few very long ones (their blocks take no other rows, or
do), against the oracle and the launched sweeps."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


def rows(n, lengths, seed):
    rng = np.random.default_rng(seed)
    u, v = [np.arange(n)], [np.arange(n)]
    for at, d in enumerate(lengths):
        u.append(rng.choice(n, d, replace=False))
        v.append(np.full(d, at))
    key = np.unique(np.concatenate(u).astype(np.int64) * n + np.concatenate(v))
    off = np.zeros(n + 1, np.uint32)
    off[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    return off, (key % n).astype(np.uint32)


CASES = {
    "many": lambda: rows(5000, [1025 + 3 * (i % 900) for i in range(1000)] + [4096, 4097, 4500, 300, 70], 1),
    "few": lambda: rows(5000, [1025, 1500, 4096, 4097, 4500, 300, 70], 2),
    "solo": lambda: rows(60_000, [40_000, 16_385, 30_000, 100, 65], 3),
    "solo, small grid": lambda: rows(17_000, [16_900] * 12, 4),
    "as long on average": lambda: rows(40_000, [16_384] * 3, 5),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_solves(ctx, case):
    import pagerank_gb300 as pg
    xoff, xedg = CASES[case]()
    q, it = O.solve("static", None, None, *O.transpose(xoff, xedg))
    batch = pg.graphs.random_batch(xoff, xedg, 30, 90, seed=2)
    yoff, yedg = pg.graphs.apply_batch(xoff, xedg, *batch)
    yt = O.transpose(yoff, yedg)
    g = pg.Graph(ctx, *yt, yoff, yedg)
    for mode in ("static", "naive_dynamic", "dynamic_traversal", "dynamic_frontier", "prune_dynamic_frontier"):
        want, it = O.solve(mode, yoff, yedg, *yt, *batch, q=q)
        for kw in ({}, {"loop": pg.LOOP_GRAPH}):
            r, res = pg.solve(ctx, g, pg.MODES[mode], batch[:2], batch[2:], q, pg.options(**kw))
            assert res["iterations"] == it and np.array_equal(r, want), (mode, kw)
    want, b = pg.solve(ctx, g, pg.STATIC, opts=pg.options(precision=pg.FP32_REFINE, loop=pg.LOOP_GRAPH))
    r, a = pg.solve(ctx, g, pg.STATIC, opts=pg.options(precision=pg.FP32_REFINE))
    assert a["iterations"] == b["iterations"] and np.array_equal(r, want)
    g.close()


@pytest.mark.parametrize("side", ["in", "out"])
@pytest.mark.parametrize("case", sorted(CASES))
def test_weighted(ctx, case, side):
    import pagerank_gb300 as pg
    import torch
    from pagerank_gb300 import autograd as A
    xoff, xedg = CASES[case]()
    n, m = len(xoff) - 1, len(xedg)
    xtoff, xtedg, xtdat = O.transpose(xoff, xedg)
    if side == "out":   # the long rows are out-rows
        xoff, xedg, (xtoff, xtedg, _) = xtoff, xtedg, (xoff, xedg, None)
        xtdat = np.diff(xoff.astype(np.int64)).astype(np.uint32)
    g = pg.Graph(ctx, xtoff, xtedg, xtdat, xoff, xedg, validate=True)
    gen = torch.Generator(device="cuda").manual_seed(5)
    w = 0.5 + torch.rand(m, generator=gen, device="cuda")
    goal = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) - 0.5
    A.set_weights(ctx, g, w)
    got = []
    for loop in (pg.LOOP_AUTO, pg.LOOP_HOST):
        o = pg.options(tolerance=1e-14, max_iterations=400, loop=loop)
        r, _ = A.solve_weighted(ctx, g, opts=o)
        got.append([r, A.adjoint(ctx, g, r, goal, opts=o)["grad_w"]])
    for a, b in zip(*got):   # rows of up to 40,000 terms in another order: 4e4 * 2^-53 / (1 - 0.85) < 3e-11
        assert float((a - b).abs().max()) <= 3e-11 * float(b.abs().max())
    # the same fixed points from the definition, each iterated to a step of 1e-14
    u = torch.repeat_interleave(torch.arange(n, device="cuda"), torch.from_numpy(np.diff(xoff.astype(np.int64))).cuda())
    v = torch.from_numpy(xedg.astype(np.int64)).cuda()
    zero = lambda: torch.zeros(n, dtype=torch.float64, device="cuda")  # noqa: E731
    s = zero().index_add_(0, u, w.double())
    p = w.double() / s[u]
    r, lam = zero() + 1 / n, goal.clone()
    for _ in range(400):
        r = 0.15 / n + 0.85 * zero().index_add_(0, v, p * r[u])
        lam = goal + 0.85 * zero().index_add_(0, u, p * lam[v])
    mean = zero().index_add_(0, u, p * lam[v])
    grad = 0.85 * r[u] * (lam[v] - mean[u]) / s[u]
    for a, b in zip(got[0], (r, grad)):
        assert float((a - b).abs().max()) <= 3e-11 * float(b.abs().max()) + 1.2e-13
    g.close()
