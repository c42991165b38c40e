"""Calls one of whose device allocations fails: each returns out of memory or
the right result, and leaves nothing half built for the next call to use."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu
ENOMEM, ESTATE = 2, 6


@pytest.fixture(scope="module")
def pg():
    import pagerank_gb300
    return pagerank_gb300


def failing(pg, call, most=200):
    """call() with its 1st, 2nd, ... allocation failing, until it makes no more:
    yields the error (None: it went through all the same)."""
    for nth in range(1, most):
        pg.selftest_fail_alloc(nth)
        try:
            call()
            error = None
        except pg.PrxError as e:
            error = e
        finally:
            left = pg.selftest_fail_alloc(0)
        if left:
            assert error is None
            return
        assert error is None or error.status == ENOMEM, error
        yield error
    raise AssertionError("more allocations than expected")


def graph(pg, ctx, kind, seg_shift=0):
    xoff, xedg = {"rmat": lambda: pg.graphs.rmat(12, 16, seed=3),
                  "web": lambda: pg.graphs.weblike(3001, dmax=900, window=512, seed=9)}[kind]()
    xt = O.transpose(xoff, xedg)
    if seg_shift:
        return pg.Graph.from_csr64(ctx, xt[0], xt[1], xt[2], xoff, xedg, seg_shift=seg_shift)
    return pg.Graph(ctx, *xt, xoff, xedg)


@pytest.mark.parametrize("seg_shift", [0, 10])
@pytest.mark.parametrize("kind", ["rmat", "web"])
def test_set_weights(pg, ctx, kind, seg_shift):
    import torch
    from pagerank_gb300 import autograd as A
    g = graph(pg, ctx, kind, seg_shift)
    n, m = g.size()
    gen = torch.Generator(device="cuda").manual_seed(7)
    w = 0.5 + torch.rand(m, generator=gen, device="cuda")
    goal = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)

    def gradients(x):
        r, _ = A.solve_weighted(ctx, x)
        return [r, A.adjoint(ctx, x, r, goal)["grad_w"]]

    A.set_weights(ctx, g, w)
    want = gradients(g)
    g.close()
    failed = 0
    for spent in (False, True):   # on a graph without weights and on one whose weights a batch has dropped
        def fresh():
            x = graph(pg, ctx, kind, seg_shift)
            if spent:
                A.set_weights(ctx, x, 2 * w)
                edge, none = (np.zeros(1, np.uint32), x.download64()[1][:1]), (np.zeros(0, np.uint32),) * 2
                x.apply_batch(*edge, *none)
                x.apply_batch(*none, *edge)
            return x

        x = fresh()
        for error in failing(pg, lambda: A.set_weights(ctx, x, w)):
            if error:
                failed += 1
                with pytest.raises(pg.PrxError) as e:   # no weights rather than some of them
                    A.solve_weighted(ctx, x)
                assert e.value.status == ESTATE
                A.set_weights(ctx, x, w)
            # without its row plan the adjoint is summed in another order (up to 4096 terms a
            # row, 1 / (1 - 0.85) of it over the iterations: 4096 * 2^-53 / 0.15 < 1e-11)
            for a, b in zip(gradients(x), want):
                assert torch.equal(a, b) if error else float((a - b).abs().max()) <= 1e-11 * float(b.abs().max())
            x.close()
            x = fresh()
        x.close()
    assert failed >= 8


@pytest.mark.parametrize("mode", ["static", "naive_dynamic", "prune_dynamic_frontier", "refine"])
@pytest.mark.parametrize("kind", ["rmat", "web"])
def test_solve_without_row_plans(pg, ctx, kind, mode):
    # all that a second graph's solve allocates is what it can do without
    kw = {"precision": pg.FP32_REFINE} if mode == "refine" else {}
    m = pg.MODES["static" if mode == "refine" else mode]
    ins = (np.array([5, 9], np.uint32), np.array([7, 3], np.uint32))
    first = graph(pg, ctx, kind)
    q = np.full(first.size()[0], 1.0 / first.size()[0])

    def solve(x):
        return pg.solve(ctx, x, m, None, ins if m > 1 else None, q if m else None, pg.options(**kw))

    want, res = solve(first)
    pg.solve(ctx, first, pg.STATIC, opts=pg.options(hot_sources=1000))   # the hot copy's buffers
    first.close()
    passed = 0
    got = []
    x = graph(pg, ctx, kind)
    for error in failing(pg, lambda: got.append(solve(x))):
        assert error is None
        passed += 1
        r, again = got.pop()
        assert again["iterations"] == res["iterations"] and np.array_equal(r, want)
        r, again = solve(x)
        assert again["iterations"] == res["iterations"] and np.array_equal(r, want)
        x.close()
        x = graph(pg, ctx, kind)
    assert passed >= 2
    x.close()


def test_weighted_solve_without_row_plans(pg, ctx):
    import torch
    from pagerank_gb300 import autograd as A
    w = None
    want, passed = None, 0
    for round in (0, 1):
        x = graph(pg, ctx, "rmat")
        if w is None:
            w = 0.5 + torch.rand(x.size()[1], generator=torch.Generator(device="cuda").manual_seed(7), device="cuda")
        A.set_weights(ctx, x, w)
        if round == 0:
            want = A.solve_weighted(ctx, x)[0]
            x.close()
            continue
        got = []
        for error in failing(pg, lambda: got.append(A.solve_weighted(ctx, x)[0])):
            assert error is None
            passed += 1
            assert float((got.pop() - want).abs().max()) <= 1e-11 * float(want.max())   # as above
            x.close()
            x = graph(pg, ctx, "rmat")
            A.set_weights(ctx, x, w)
        x.close()
    assert passed >= 2


def test_apply_batch_without_its_layout(pg, ctx):
    xoff, xedg = pg.graphs.weblike(3001, dmax=900, window=512, seed=9)
    batch = pg.graphs.random_batch(xoff, xedg, 40, 100, seed=2)
    yoff, yedg = pg.graphs.apply_batch(xoff, xedg, *batch)
    want, it = O.solve("static", None, None, *O.transpose(yoff, yedg))
    opts = pg.options(chunk_vertices=1000, hot_sources=200)

    def fresh():
        x = graph(pg, ctx, "web")
        pg.pagerank_static(ctx, x, opts)   # builds the layout that a batch carries on
        return x

    x, passed = fresh(), 0
    for error in failing(pg, lambda: x.apply_batch(*batch)):
        if error is None:
            passed += 1
            r, res = pg.pagerank_static(ctx, x, opts)
            assert res["iterations"] == it and np.array_equal(r, want)
        x.close()
        x = fresh()
    assert passed >= 3   # the layout's offsets, ids and scan
    x.close()


@pytest.mark.parametrize("vectors", [5, 24, 64])
@pytest.mark.parametrize("refine", [False, True])
@pytest.mark.parametrize("kind", ["hubs", "web"])
def test_personalized_solve(pg, kind, refine, vectors):
    xoff, xedg = {"hubs": lambda: pg.graphs.rmat(12, 48, a=0.7, b=0.1, c=0.1, seed=3),   # rows of several segments
                  "web": lambda: pg.graphs.weblike(3001, dmax=900, window=512, seed=9)}[kind]()
    n = len(xoff) - 1
    xt = O.transpose(xoff, xedg)
    rng = np.random.default_rng(4)
    seeds = [rng.integers(0, n, 1 + k % 5) for k in range(vectors)]
    opts = pg.options(tolerance=1e-9, precision=pg.FP32_REFINE if refine else pg.FP64)

    def fresh():
        c = pg.Context(0)
        return c, pg.Graph(c, *xt, xoff, xedg)

    def solve(c, g):
        return pg.solve_ppr_batched(c, g, seeds, opts)

    c, g = fresh()
    want, res = solve(c, g)
    passed, failed, got = 0, 0, []
    c.close()
    g.close()
    c, g = fresh()
    for error in failing(pg, lambda: got.append(solve(c, g))):
        if error is None:
            passed += 1
            r, again = got.pop()
            assert np.array_equal(r, want) and again["iterations"] == res["iterations"]
        else:
            failed += 1
        r, again = solve(c, g)
        assert np.array_equal(r, want) and again["iterations"] == res["iterations"]
        g.close()
        c.close()
        c, g = fresh()
    # the length list and its sort, the partial rows and where they start (graphs with
    # long rows), and the pairs of the FP32 sweeps
    long_rows = bool((np.diff(xt[0].astype(np.int64)) > 64).any())
    assert passed >= 2 + 2 * long_rows + (refine and vectors < 64), (passed, failed)
    g.close()
    c.close()


@pytest.mark.parametrize("seg_shift", [0, 10])
def test_apply_batch_is_all_or_nothing(pg, ctx, seg_shift):
    xoff, xedg = pg.graphs.rmat(12, 16, seed=3)
    old, it_old = O.solve("static", None, None, *O.transpose(xoff, xedg))
    batch = pg.graphs.random_batch(xoff, xedg, 40, 100, seed=2)
    yoff, yedg = pg.graphs.apply_batch(xoff, xedg, *batch)
    want, it = O.solve("static", None, None, *O.transpose(yoff, yedg))

    def holds(x, ranks, iterations):
        for kw in ({}, {"loop": pg.LOOP_GRAPH}):
            r, res = pg.pagerank_static(ctx, x, pg.options(**kw))
            assert res["iterations"] == iterations and np.array_equal(r, ranks)

    x, failed = graph(pg, ctx, "rmat", seg_shift), 0
    for error in failing(pg, lambda: x.apply_batch(*batch)):
        if error:
            failed += 1
            holds(x, old, it_old)     # unchanged, and the batch still applies
            x.apply_batch(*batch)
        holds(x, want, it)
        x.close()
        x = graph(pg, ctx, "rmat", seg_shift)
    assert failed >= 8
    x.close()
