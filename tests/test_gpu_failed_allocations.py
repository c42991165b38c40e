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
            assert all(torch.equal(a, b) for a, b in zip(gradients(x), want))
            x.close()
            x = fresh()
        x.close()
    assert failed >= 8
