"""Ranks that the integer adder does not take (zero, subnormal, tiny, negative,
huge, infinite, NaN) among those that it does, in rows of every class: the sums of
every path are the oracle's, in the cooperative loop and in the launched sweeps by
row, by words and by chunk.

The library divides by a reciprocal, so the contribution of an infinite rank is
NaN (inf - inf in its remainder) where a division would leave infinity; and a NaN
change does not end its loop, where the oracle's maximum passes it over.  Infinite
and NaN ranks are therefore compared with the oracle's sums of NaN ranks after one
iteration, and the paths with one another after more."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

# rows of the LOW bound and its remainders, of MID and of HIGH (in-degrees over
# 1024 go by block in the cooperative loop, over 4096 in the launched one)
LENGTHS = [1, 2, 3, 4, 5, 33, 63, 64, 65, 66, 95, 128, 129, 160, 161, 193, 225, 255, 256, 257, 300, 513, 1024, 1025, 1100,
           4096, 4097, 4400]
VALUES = {"zero": 0.0, "negative zero": -0.0, "subnormal": 5e-324, "tiny": 1e-290, "negative": -1e-3, "huge": 1e300,
          "infinite": np.inf, "nan": np.nan}


def by_rows(n, lengths, seed):
    rng = np.random.default_rng(seed)
    u, v = [np.arange(n)], [np.arange(n)]
    for at, d in enumerate(lengths):
        u.append(rng.choice(np.delete(np.arange(n), at), d - 1, replace=False))
        v.append(np.full(d - 1, at))
    key = np.unique(np.concatenate(u).astype(np.int64) * n + np.concatenate(v))
    off = np.zeros(n + 1, np.uint32)
    off[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    return off, (key % n).astype(np.uint32)


GRAPHS = {"rows": lambda pg: by_rows(4500, LENGTHS, 3),                              # LOW rows of one id
          "even": lambda pg: pg.graphs.weblike(5003, dmax=900, window=512, seed=9)}  # laid out by words when launched


def same(a, b):
    nan = np.isnan(a) & np.isnan(b)
    return np.array_equal(a.view(np.uint64)[~nan], b.view(np.uint64)[~nan])


@pytest.mark.parametrize("spread", [97, 2, 1])   # a few of the sources, every other one, all
@pytest.mark.parametrize("value", sorted(VALUES))
@pytest.mark.parametrize("kind", sorted(GRAPHS))
def test_sums_equal_the_oracle(ctx, kind, value, spread):
    import pagerank_gb300 as pg
    xoff, xedg = GRAPHS[kind](pg)
    n = len(xoff) - 1
    xt = O.transpose(xoff, xedg)
    q = np.random.default_rng(1).random(n) / n
    q[::spread] = VALUES[value]
    e, one = np.zeros(0, np.uint32), np.arange(0, n, 7, dtype=np.uint32)
    g = pg.Graph(ctx, *xt, xoff, xedg, validate=True)
    paths = [{}, {"int_adds": -1}, {"loop": pg.LOOP_GRAPH}, {"loop": pg.LOOP_GRAPH, "hot_sources": -1},
             {"loop": pg.LOOP_GRAPH, "int_adds": -1}, {"chunk_vertices": 1000}]
    finite = np.isfinite(VALUES[value])
    for mode in ("naive_dynamic", "dynamic_frontier", "prune_dynamic_frontier"):
        ins = (e, e) if mode == "naive_dynamic" else (one, one)
        for cap in (1, 3):
            if finite or (cap == 1 and mode == "naive_dynamic"):
                want, it = O.solve(mode, xoff, xedg, *xt, e, e, *ins, q=np.where(np.isfinite(q), q, np.nan),
                                   opts=O.options(max_iterations=cap))
            else:
                want, res = pg.solve(ctx, g, pg.MODES[mode], None, ins, q,
                                     pg.options(max_iterations=cap, loop=pg.LOOP_HOST, int_adds=-1))
                it = res["iterations"]
            for kw in paths:
                r, res = pg.solve(ctx, g, pg.MODES[mode], None, ins, q, pg.options(max_iterations=cap, **kw))
                assert res["iterations"] == it and same(r, want), (mode, cap, kw)
    g.close()
