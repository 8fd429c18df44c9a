"""Contraction by ranges (integer weights, at least 2^24 entries): large communities over few and many
next-level ids, member rows longer than a piece's limit, ranges longer than a folded slice, self-loop
weights, a batch whose graphs have their own id ranges. Exact: partition, community count, modularity
and the first contracted graph's row sums and weights."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(lv, n, pairs, blocks, hubs, seed, weights="unit"):
    """`blocks` planted communities (9 pairs of 10 inside), `hubs` vertices joined to a third of all."""
    rng = np.random.default_rng(seed)
    size = n // blocks
    u = rng.integers(0, n, pairs)
    inside = rng.random(pairs) < 0.9
    v = np.where(inside, (u // size) * size + rng.integers(0, size, pairs), rng.integers(0, n, pairs))
    v = np.minimum(v, n - 1)
    h = rng.integers(0, n, hubs)
    u = np.concatenate([u, np.repeat(h, n // 3), np.arange(n)])
    v = np.concatenate([v, rng.integers(0, n, hubs * (n // 3)), (np.arange(n) + 1) % n])
    w = rng.integers(1, 6, u.size).astype(np.float32) if weights == "int" else None
    return lv.graphs.canonical_from_pairs(u, v, w)


@pytest.mark.parametrize("n,pairs,blocks,hubs,weights", [(40_000, 9_400_000, 20, 3, "unit"), (150_000, 10_800_000, 400, 2, "int")])
def test_single(n, pairs, blocks, hubs, weights, lv, oracle):
    g = _graph(lv, n, pairs, blocks, hubs, 5, weights)
    assert g.E >= 1 << 24
    o = oracle.Oracle(g, mode=oracle.SORT)
    o.louvain()
    eng = lv.Engine(0)
    best, q, st = eng.run_graph(g)
    np.testing.assert_array_equal(best, o.best())
    assert q == o.modularity and st.n_communities == o.n_best
    c = eng.community(g)
    c.optimization_run()
    comm, _tot = c.partition()
    ids = np.unique(comm)
    new = np.searchsorted(ids, comm)
    want = np.bincount(new[g.src()].astype(np.int64) * ids.size + new[g.col], weights=g.weights_or_ones.astype(np.float64),
                       minlength=ids.size * ids.size) if ids.size <= 4000 else None
    c.aggregation_run(True)
    row, col, w, k = c.graph()
    np.testing.assert_array_equal(k, np.bincount(new[g.src()], weights=g.weights_or_ones.astype(np.float64), minlength=ids.size))
    src = np.repeat(np.arange(ids.size), np.diff(row))
    key = src.astype(np.int64) * ids.size + col
    assert np.unique(key).size == key.size  # one entry per pair
    if want is not None:
        got = np.zeros(ids.size * ids.size)
        got[key] = w
        np.testing.assert_array_equal(got, want)
    eng.close()


def test_batch(lv, oracle):
    batch = importlib.import_module("louvain-fast-move-cuda_b200.batch")
    gs = [_graph(lv, n, p, b, 1, n) for n, p, b in ((30_001, 4_000_000, 15), (9_000, 100_000, 9), (50_000, 6_400_000, 60))]
    offs, row, col, _ = batch.pack(gs)
    assert col.size >= 1 << 24
    eng = lv.Engine(0)
    out, q, k, _ = eng.run_batch(offs, row, col)
    eng.close()
    for i, g in enumerate(gs):
        o = oracle.Oracle(g, mode=oracle.SORT)
        o.louvain()
        np.testing.assert_array_equal(out[offs[i]:offs[i + 1]], o.best())
        assert q[i] == o.modularity and k[i] == o.n_best
