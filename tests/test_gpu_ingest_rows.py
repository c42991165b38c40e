"""Graph ingest at the row lengths where the row sort changes hands (8 lanes, a
warp's registers, a block's shared memory, the radix sort), with and without
duplicates, in both directions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGES = [0, 1, 2, 7, 8, 9, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 2049]
LONG = [16383, 16384, 16385, 20000, 40001]


def csr(n, u, v):
    key = np.unique(u.astype(np.uint64) * n + v)
    off = np.searchsorted(key, np.arange(n + 1, dtype=np.uint64) * n)
    return off.astype(np.uint32), (key % n).astype(np.uint32)


@pytest.mark.parametrize("loops", [False, True])
@pytest.mark.parametrize("dups", [False, True])
@pytest.mark.parametrize("lengths,n", [(EDGES, 3001), (LONG[:3] + EDGES, 50001), (LONG, 41003), ([], 5), ([1], 1)])
def test_rows(ctx, lengths, n, dups, loops):
    import pagerank_gb300 as pg
    rng = np.random.default_rng(len(lengths) + n)
    u, v = [np.zeros(0, np.uint32)], [np.zeros(0, np.uint32)]
    for k in lengths:
        a = rng.integers(0, n)
        b = rng.permutation(n)[:k].astype(np.uint32)
        if dups and k:  # same length, a fifth of it repeated
            b[rng.integers(0, k, k // 5)] = b[0]
        u.append(np.full(k, a, np.uint32))
        v.append(b)
    u, v = np.concatenate(u), np.concatenate(v)
    p = rng.permutation(len(u))
    uu, vv = (u, v)
    if loops:
        i = np.arange(n, dtype=np.uint32)
        uu, vv = np.concatenate([u, i]), np.concatenate([v, i])
    want, back = csr(n, uu, vv), csr(n, vv, uu)
    for fwd in (True, False):   # the long rows are the out-rows, then the in-rows
        g = pg.Graph.from_edges(ctx, n, *((u[p], v[p]) if fwd else (v[p], u[p])), self_loops=loops)
        xoff, xedg, xtoff, xtedg, deg = g.download()
        for got, ref in (((xoff, xedg), want if fwd else back), ((xtoff, xtedg), back if fwd else want)):
            assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
        assert np.array_equal(deg, np.diff((want if fwd else back)[0]))
        g.close()
