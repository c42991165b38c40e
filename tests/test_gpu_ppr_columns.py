"""Batched personalized PageRank at every stored row width: a vector's ranks
after a fixed number of sweeps do not depend on the vectors beside it, so the
first k columns of a 64-vector solve must come out bit for bit from a solve of
k vectors (rows of 8 to 64 columns, short and long rows, ragged batches)."""
import numpy as np
import pytest

from oracle import ppr_oracle as PO
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pg():
    import pagerank_gb300
    return pagerank_gb300


GRAPHS = {
    "hubs": lambda pg: pg.graphs.rmat(13, 48, a=0.7, b=0.1, c=0.1, seed=3),   # rows over several segments
    "web": lambda pg: pg.graphs.weblike(7001, dmax=900, window=512, seed=9),
    "33": lambda pg: pg.graphs.grid(6, seed=2),
}


@pytest.mark.parametrize("kind", sorted(GRAPHS))
@pytest.mark.parametrize("refine", [False, True])
def test_columns_independent_of_width(pg, ctx, kind, refine):
    xoff, xedg = GRAPHS[kind](pg)
    n = len(xoff) - 1
    xt = O.transpose(xoff, xedg)
    g = pg.Graph(ctx, *xt, xoff, xedg)
    rng = np.random.default_rng(4)
    seeds = [rng.integers(0, n, 1 + k % 5) for k in range(64)]
    opts = pg.options(tolerance=0.0, max_iterations=5, precision=pg.FP32_REFINE if refine else pg.FP64)
    full, _ = pg.solve_ppr_batched(ctx, g, seeds, opts)
    if not refine:
        want, _ = PO.jacobi(*xt, seeds, tol=0.0, max_iter=5)
        assert np.abs(full - want).max() <= 1e-13
    for k in (1, 7, 8, 9, 16, 17, 24, 25, 32, 33, 48, 49):
        got, _ = pg.solve_ppr_batched(ctx, g, seeds[:k], opts)
        assert np.array_equal(got, full[:, :k]), k
    g.close()
