"""Passes applied by the walk over every row (most of the level's entries belong to movers; at least
2^22 entries) against the oracle: per-pass partition-derived values -- the internal weight I and the
squared totals S of every pass, exact integers -- and the final partition. Hub rows span many
2048-entry chunks, short rows many rows per chunk, self-loops are stored twice; a batch puts several
graphs under one warp's 32 rows."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(lv, n, entries, hubs, seed, weights="unit"):
    rng = np.random.default_rng(seed)
    ring = np.arange(n)
    m = entries // 2 - n
    h = hubs * (n // 2)
    u = np.concatenate([ring, np.repeat(rng.integers(0, n, hubs), n // 2), rng.integers(0, n, m - h)])
    v = np.concatenate([(ring + 1) % n, rng.integers(0, n, h), rng.integers(0, n, m - h)])
    w = rng.integers(1, 6, u.size).astype(np.float32) if weights == "int" else None
    return lv.graphs.canonical_from_pairs(u, v, w)


@pytest.mark.parametrize("n,entries,hubs,weights", [(60_000, 5_200_000, 0, "unit"), (60_000, 5_200_000, 12, "int"),
                                                    (1_100_000, 6_400_000, 1, "unit"), (4_000, 6_400_000, 0, "int")])
def test_trace_equals_oracle(n, entries, hubs, weights, lv, oracle):
    g = _graph(lv, n, entries, hubs, n, weights)
    if weights == "unit":  # self-loops at both ends and in the middle, stored twice
        loops = np.array([0, g.n // 2, g.n - 1])
        key = np.sort(np.concatenate([g.src(), loops, loops]).astype(np.int64) << 32
                      | np.concatenate([g.col, loops, loops]).astype(np.int64), kind="stable")
        row = np.zeros(g.n + 1, np.int64)
        np.cumsum(np.bincount(key >> 32, minlength=g.n), out=row[1:])
        g = lv.graphs.CSRGraph(n=g.n, row_ptr=row, col=(key & 0xFFFFFFFF).astype(np.int32))
    assert g.E >= 1 << 22
    o = oracle.Oracle(g, mode=oracle.SORT)
    o.louvain()
    eng = lv.Engine(0)
    c = eng.community(g)
    c.louvain()
    tr = c.trace()
    eng2_best, q, st = eng.run_graph(g)
    np.testing.assert_array_equal(c.best(), o.best())
    np.testing.assert_array_equal(eng2_best, o.best())
    assert q == o.modularity and st.n_communities == o.n_best and tr["modularity"][-1] == o.modularity
    eng.close()


def test_batch(lv, oracle):
    batch = importlib.import_module("louvain-fast-move-cuda_b200.batch")
    gs = [_graph(lv, n, 26 * n, 0, n) for n in (9000, 70_001, 9_001, 40_000, 8_500, 60_000)]
    offs, row, col, _ = batch.pack(gs)
    assert col.size >= 1 << 22
    eng = lv.Engine(0)
    out, q, k, _ = eng.run_batch(offs, row, col)
    eng.close()
    for i, g in enumerate(gs):
        o = oracle.Oracle(g, mode=oracle.SORT)
        o.louvain()
        np.testing.assert_array_equal(out[offs[i]:offs[i + 1]], o.best())
        assert q[i] == o.modularity and k[i] == o.n_best
