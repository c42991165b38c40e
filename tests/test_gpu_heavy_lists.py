"""Edge lists of 2^23 entries, most of them in a few very long rows or repeated: both
CSRs against numpy, also when an allocation fails, and ids out of range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
M, N = 1 << 23, 70_000


def draw(kind):
    rng = np.random.default_rng(3)
    any_, hub = rng.integers(0, N, M, dtype=np.int64), rng.integers(0, 40, M, dtype=np.int64)
    part = rng.random(M) < {"most from hubs": 0.85, "half from hubs": 0.5}.get(kind, 0)
    return {"from hubs": (hub, any_), "to hubs": (any_, hub), "one edge": (np.full(M, 7), np.full(M, N - 1)),
            "pairs": (hub, rng.integers(0, 40, M, dtype=np.int64)),
            "most from hubs": (np.where(part, hub, rng.integers(0, N, M)), any_),
            "half from hubs": (np.where(part, hub, rng.integers(0, N, M)), any_),
            "one short": (hub[:-1], any_[:-1])}[kind]


@pytest.mark.parametrize("loops", [False, True])
@pytest.mark.parametrize("kind", ["from hubs", "to hubs", "one edge", "pairs", "most from hubs", "half from hubs",
                                  "one short"])
def test_csr(ctx, kind, loops):
    import pagerank_gb300 as pg
    import torch
    u, v = draw(kind)
    key = np.unique(np.concatenate([u * N + v] + ([np.arange(N) * (N + 1)] if loops else [])))
    du, dv = (torch.from_numpy(x.astype(np.int32)).cuda() for x in (u, v))
    for nth in (0, 1, 3, 6, 8):   # 0: none fails
        pg.selftest_fail_alloc(nth)
        try:
            g = pg.Graph.from_device_edges(ctx, N, du, dv, self_loops=loops)
        except pg.PrxError as e:
            assert nth and e.status == 2
            continue
        finally:
            pg.selftest_fail_alloc(0)
        off, edg, xt, tedg, deg = g.download()
        assert np.array_equal(edg, key % N) and np.array_equal(off, np.searchsorted(key // N, np.arange(N + 1)))
        back = np.sort(key % N * N + key // N)
        assert np.array_equal(tedg, back % N) and np.array_equal(xt, np.searchsorted(back // N, np.arange(N + 1)))
        assert np.array_equal(deg, np.diff(off))
        g.close()
    du[M // 3] = N
    with pytest.raises(pg.PrxError, match="out of range"):
        pg.Graph.from_device_edges(ctx, N, du, dv, self_loops=loops)
