"""What a batched personalized solve reports and keeps: the kernel that builds the
FP32 sweeps' pairs of edges runs in every such call and is counted with it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vectors", [5, 40])
def test_pairs_are_counted(ctx, vectors):
    import pagerank_gb300 as pg
    g = pg.Graph.from_out_csr(ctx, *pg.graphs.rmat(12, 16, seed=3))
    seeds = [np.array([k]) for k in range(vectors)]

    def launches(precision):
        return pg.solve_ppr_batched(ctx, g, seeds, pg.options(max_iterations=0, precision=precision))[1]["kernel_launches"]

    fp64 = launches(pg.FP64)                                # initial ranks, control block, output
    assert fp64 == 3 and launches(pg.FP32_REFINE) == fp64 + 1
    g.close()
