"""FP32 refinement as one cooperative kernel (the default of Static and ND on
small and medium graphs): ranks, iterations and refinements of the launched loop
bit for bit, where rows and iteration caps meet their edges."""
import numpy as np
import pytest

from oracle import pyoracle as O
from test_gpu_persist import CASES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", sorted(CASES))
def test_equals_launched_loop(ctx, case):
    import pagerank_gb300 as pg
    xoff, xedg = CASES[case](pg)
    g = pg.Graph(ctx, *O.transpose(xoff, xedg), xoff, xedg)
    q = np.random.default_rng(1).random(len(xoff) - 1)
    q /= q.sum()
    for mode, start in ((pg.STATIC, None), (pg.NAIVE_DYNAMIC, q)):
        for kw in ({}, {"max_iterations": 0}, {"max_iterations": 1}, {"max_iterations": 2}, {"max_iterations": 3},
                   {"max_iterations": 20}, {"tolerance": 1e-4}, {"tolerance": 1e-13}):
            want, b = pg.solve(ctx, g, mode, q=start, opts=pg.options(precision=pg.FP32_REFINE, loop=pg.LOOP_GRAPH, **kw))
            r, a = pg.solve(ctx, g, mode, q=start, opts=pg.options(precision=pg.FP32_REFINE, **kw))
            assert np.array_equal(r, want), (mode, kw)
            for key in ("iterations", "refinements", "last_delta", "edges_processed"):
                assert a[key] == b[key], (mode, kw, key)
    g.close()


@pytest.mark.parametrize("case", sorted(CASES))
def test_same_bits_without_integer_adds(ctx, case):
    import pagerank_gb300 as pg
    xoff, xedg = CASES[case](pg)
    g = pg.Graph(ctx, *O.transpose(xoff, xedg), xoff, xedg)
    want, b = pg.solve(ctx, g, pg.STATIC, opts=pg.options(precision=pg.FP32_REFINE))
    r, a = pg.solve(ctx, g, pg.STATIC, opts=pg.options(precision=pg.FP32_REFINE, int_adds=-1))
    assert np.array_equal(r, want) and a["iterations"] == b["iterations"]
    g.close()
