"""Batched personalized PageRank on rows of 4 to 9 segments of 512 in-edges around the
line where blocks combine them, and of up to 80: the same bits as the same columns in
blocks of other widths, and the Jacobi iteration in float64."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


def graph(ctx):
    import pagerank_gb300 as pg
    n = 42_000
    rng = np.random.default_rng(1)
    lengths = [2047, 2048, 2049, 2111, 2112, 4096, 15_872, 15_873, 16_385, 40_961, 65]
    u = np.concatenate([rng.choice(n, d, replace=False) for d in lengths] + [rng.integers(0, n, 2 * n), np.arange(n)])
    v = np.concatenate([np.full(d, 100 + i) for i, d in enumerate(lengths)] + [rng.integers(0, n, 2 * n), np.arange(n)])
    key = np.unique(u.astype(np.int64) * n + v)
    off = np.zeros(n + 1, np.uint32)
    off[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    edg = (key % n).astype(np.uint32)
    return n, key, off, pg.Graph(ctx, *O.transpose(off, edg), off, edg)


@pytest.mark.parametrize("cols", [1, 8, 16, 24, 32, 48, 64])
def test_rows(ctx, cols):
    import pagerank_gb300 as pg
    n, key, off, g = graph(ctx)
    seeds = [np.array([(7919 * k + i) % n for i in range(1 + k % 3)], np.uint32) for k in range(cols)]
    src, dst, deg = key // n, key % n, np.diff(off.astype(np.int64))
    for prec in (pg.FP64, pg.FP32_REFINE):
        opts = pg.options(precision=prec, tolerance=1e-12, max_iterations=500)
        r, res = pg.solve_ppr_batched(ctx, g, seeds, opts)
        r = np.asarray(r).reshape(n, cols)
        for k in sorted({0, cols // 2, cols - 1}):
            t = np.bincount(seeds[k], minlength=n) / len(seeds[k])
            want = t.copy()
            for _ in range(260):   # 0.85^260 < 5e-19
                want = 0.15 * t + 0.85 * np.bincount(dst, want[src] / deg[src], n)
            # a step below 1e-12 leaves at most 0.85/0.15 * 1e-12 a vertex of its column in the
            # largest norm times the largest row's part; rounding is far below
            assert np.abs(r[:, k] - want).max() <= 1e-11 + 1e-9 * want.max(), (prec, k)
        one, _ = pg.solve_ppr_batched(ctx, g, seeds[:1], pg.options(precision=prec, tolerance=0.0, max_iterations=20))
        all_, _ = pg.solve_ppr_batched(ctx, g, seeds, pg.options(precision=prec, tolerance=0.0, max_iterations=20))
        if prec == pg.FP64:
            assert np.array_equal(np.asarray(one).reshape(n), np.asarray(all_).reshape(n, cols)[:, 0])
    g.close()


@pytest.mark.parametrize("prec, cols", [("FP64", 5), ("FP64", 64), ("FP32_REFINE", 5), ("FP32_REFINE", 64)])
def test_rows_without_memory_for_their_parts(ctx, prec, cols):
    import pagerank_gb300 as pg
    opts = pg.options(precision=getattr(pg, prec), tolerance=0.0, max_iterations=20)
    _, _, _, g = graph(ctx)
    seeds = [np.array([7919 * k % 42_000], np.uint32) for k in range(cols)]
    want = pg.solve_ppr_batched(ctx, g, seeds, opts)[0]
    g.close()
    same = 0
    for nth in range(1, 16):
        c = pg.Context(0)
        g = graph(c)[3]
        pg.selftest_fail_alloc(nth)
        try:
            r = pg.solve_ppr_batched(c, g, seeds, opts)[0]
            assert np.array_equal(r, want), nth
            same += 1
        except pg.PrxError:
            pass
        finally:
            pg.selftest_fail_alloc(0)
        g.close()
        c.close()
    assert same >= 3   # the partial rows, their list and the list of lengths
