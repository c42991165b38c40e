"""Probabilities and weight sums of out-rows of every length around the classes'
edges, by one lane a row and by eight (average row of four edges and more), against
float64 sums, with and without rows past 1024."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

CASES = {  # out-row lengths, self-loop included
    "one lane": [1, 2, 3] * 50 + [7, 8, 9],
    "eight lanes": list(range(1, 65)) * 2 + [31, 33],
    "longer": list(range(1, 70)) + [127, 128, 1023, 1024, 1025, 1500],
    "long in short": [1] * 3000 + [64, 65, 1024, 1025, 4096, 4097],
    "many long": [1025 + i % 300 for i in range(930)] + [5, 64, 65],
    "one row": [5],
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_probabilities(ctx, case):
    import pagerank_gb300 as pg
    import torch
    from pagerank_gb300 import autograd as A
    rng = np.random.default_rng(4)
    length = np.array(CASES[case])
    n = max(len(length), int(length.max()))
    length = np.concatenate([length, np.ones(n - len(length), int)])
    off = np.zeros(n + 1, np.uint32)
    off[1:] = np.cumsum(length)
    edg = np.concatenate([np.sort(np.append(rng.choice(np.delete(np.arange(n), v) if d > 1 else [v], d - 1, False), v))
                          for v, d in enumerate(length)]).astype(np.uint32)
    g = pg.Graph(ctx, *O.transpose(off, edg), off, edg, validate=True)
    w = (0.25 + rng.random(len(edg))).astype(np.float32)
    A.set_weights(ctx, g, torch.from_numpy(w).cuda())
    # one sweep from the uniform ranks: r1 = (1 - a)/n + (a/n) * P^T 1
    r, _ = A.solve_weighted(ctx, g, opts=pg.options(max_iterations=1))
    sums = np.add.reduceat(w.astype(np.float64), off[:-1].astype(np.int64))
    p = w / np.repeat(sums, length)
    want = 0.15 / n + 0.85 / n * np.bincount(edg, p, n)
    # both sides add up to 4097 terms twice over: 2 * 4097 * 2^-53 < 1e-12
    assert np.allclose(r.cpu().numpy(), want, rtol=1e-12, atol=0)
    g.close()
