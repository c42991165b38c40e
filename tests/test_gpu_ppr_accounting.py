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


def test_pairs_are_given_back():
    import pagerank_gb300 as pg
    import torch
    c = pg.Context(0)
    g = pg.Graph.from_out_csr(c, *pg.graphs.rmat(18, 16, seed=3))
    n, m = g.size()
    seeds = [np.array([k]) for k in range(20)]

    def free_after(precision):
        pg.solve_ppr_batched(c, g, seeds, pg.options(max_iterations=3, precision=precision))
        pg.release_cached_memory()
        return torch.cuda.mem_get_info()[0]

    # the FP32 rows stay with the context (three arrays of 64 columns), nothing of 8 bytes an edge
    kept = free_after(pg.FP64) - free_after(pg.FP32_REFINE)
    assert 8 * m > 32 << 20 and kept < 3 * 64 * 4 * n + (16 << 20)
    g.close()
    c.close()
