"""FP32 refinement on graphs whose rows average about 16 in-edges (where the LOW
sweep changes its step), with rows starting at every offset of a 32-byte sector,
whole and in source chunks, against the converged FP64 ranks."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunk", [0, 4000])
@pytest.mark.parametrize("mean", [15, 17, 40])
def test_refine_wide_rows(ctx, mean, chunk):
    import pagerank_gb300 as pg
    n, rng = 9001, np.random.default_rng(mean)
    deg = rng.integers(1, 2 * mean - 1, n)
    deg[:66] = np.arange(66) + 1
    v = np.repeat(np.arange(n), deg).astype(np.uint32)
    u = rng.integers(0, n, len(v)).astype(np.uint32)
    g = pg.Graph.from_edges(ctx, n, u, v, self_loops=True)
    xoff, xedg, xtoff, xtedg, xtdat = g.download()
    tight, _ = O.solve("static", None, None, xtoff, xtedg, xtdat, opts=O.options(tolerance=1e-17, max_iterations=400))
    opts = pg.options(precision=pg.FP32_REFINE, loop=pg.LOOP_GRAPH, chunk_vertices=chunk, hot_sources=-1)
    r, res = pg.pagerank_static(ctx, g, opts)
    # L-inf change below 1e-10 at a contraction of 0.85
    assert np.abs(r - tight).max() < 1e-10 * 0.85 / 0.15
    r2, res2 = pg.pagerank_static(ctx, g, pg.options(precision=pg.FP32_REFINE))
    assert np.array_equal(r, r2) and res["iterations"] == res2["iterations"]
    g.close()
