"""Batch tidying and application at list lengths where the key sort and the scan
change from one block to many launches, and with touched rows around the length
that is merged in pieces, against a host rebuild."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [1, 31, 32, 33, 1023, 1024, 1025, 4096, 4097, 8192, 8193, 16383, 16384, 16385, 32767, 32768, 40000]


def csr(n, u, v):
    key = np.unique(u.astype(np.uint64) * n + v)
    off = np.searchsorted(key, np.arange(n + 1, dtype=np.uint64) * n)
    return off.astype(np.uint32), (key % n).astype(np.uint32)


@pytest.mark.parametrize("count", LENGTHS)
def test_lists(ctx, count):
    import pagerank_gb300 as pg
    n = 70000
    rng = np.random.default_rng(count)
    # rows of 255 .. 1025 ids around the piece lengths, and 3 n ids at random
    long = np.concatenate([np.full(k, i * 7, np.uint32) for i, k in enumerate((255, 256, 257, 511, 512, 513, 1025))])
    u = np.concatenate([long, rng.integers(0, n, 3 * n).astype(np.uint32)])
    v = np.concatenate([rng.integers(0, n, len(long)).astype(np.uint32), rng.integers(0, n, 3 * n).astype(np.uint32)])
    i = np.arange(n, dtype=np.uint32)
    g = pg.Graph.from_edges(ctx, n, u, v, self_loops=True)
    # a raw batch with repeats: deletions of edges (and some of none), insertions (and some of edges)
    at = rng.integers(0, len(u), count)
    at[: len(long) // 2] = np.arange(min(count, len(long) // 2))
    du, dv = u[at], v[at]
    du, dv = du[du != dv], dv[du != dv]
    iu = np.where(rng.random(count) < 0.3, rng.integers(0, 7, count) * 7, rng.integers(0, n, count)).astype(np.uint32)
    iv = rng.integers(0, n, count).astype(np.uint32)
    iu[: count // 5], iv[: count // 5] = u[at][: count // 5], v[at][: count // 5]
    have = set((np.concatenate([u, i]).astype(np.uint64) * n + np.concatenate([v, i])).tolist())
    key = lambda a, b: a.astype(np.uint64) * np.uint64(n) + b
    want_d = np.unique(key(du, dv))
    want_i = np.array(sorted(k for k in set(key(iu, iv).tolist()) if k not in have), np.uint64)
    tdu, tdv, tiu, tiv = g.tidy_batch(du, dv, iu, iv)
    assert np.array_equal(key(np.asarray(tdu), np.asarray(tdv)), want_d)
    assert np.array_equal(key(np.asarray(tiu), np.asarray(tiv)), want_i)
    g.apply_batch(tdu, tdv, tiu, tiv)
    now = np.array(sorted((have - set(want_d.tolist())) | set(want_i.tolist())), np.uint64)
    nu, nv = (now // np.uint64(n)).astype(np.uint32), (now % np.uint64(n)).astype(np.uint32)
    out, back = csr(n, nu, nv), csr(n, nv, nu)
    xoff, xedg, xtoff, xtedg, deg = g.download()
    assert np.array_equal(xoff, out[0]) and np.array_equal(xedg, out[1])
    assert np.array_equal(xtoff, back[0]) and np.array_equal(xtedg, back[1])
    assert np.array_equal(deg, np.diff(out[0]))
    g.close()
