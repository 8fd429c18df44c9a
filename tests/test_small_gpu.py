"""One-launch runs of small graphs (lv_small.cuh) at the edges of what they take: vertex and entry
limits of both classes, clusters of 1 to 8 CTAs, rows that need a whole CTA's table, self-loops,
every mode and stop rule. Integer weights: partition, community count, modularity, levels, passes
and the per-pass trace equal to the oracle's / the general path's bit for bit. fp32 weights that are
multiples of 1/4 (sums exact): partitions equal, 1e-12 on Q for the order of the squared totals."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _random(lv, n, entries, hub, weights, seed):
    """n vertices, about `entries` CSR entries, vertex 0 with `hub` neighbours, some self-loops."""
    rng = np.random.default_rng(seed)
    ring = np.arange(n)
    block = rng.integers(0, max(1, n // 40), n)
    order = np.argsort(block, kind="stable")
    m = max(0, entries // 2 - n - hub)
    at = rng.integers(0, n, m)
    near = np.clip(at + rng.integers(-25, 26, m), 0, n - 1)
    u = np.concatenate([ring, np.zeros(hub, np.int64), order[at]])
    v = np.concatenate([(ring + 1) % n, rng.permutation(n)[:hub], order[near]])
    w = None
    if weights != "unit":
        w = rng.integers(1, 9, u.size).astype(np.float32) / (4.0 if weights == "float" else 1.0)
    g = lv.graphs.canonical_from_pairs(u, v, w)
    if weights == "unit" and n >= 3:  # add self-loops, stored twice as the loader does
        loops = np.unique(rng.integers(0, g.n, 5))
        src = np.concatenate([g.src(), loops, loops])
        dst = np.concatenate([g.col, loops, loops])
        key = np.sort(src.astype(np.int64) << 32 | dst.astype(np.int64), kind="stable")
        row = np.zeros(g.n + 1, np.int64)
        np.cumsum(np.bincount(key >> 32, minlength=g.n), out=row[1:])
        g = lv.graphs.CSRGraph(n=g.n, row_ptr=row, col=(key & 0xFFFFFFFF).astype(np.int32))
    return g


def _check(g, r, o):
    best, q, k = r
    np.testing.assert_array_equal(best, o.best())
    assert k == o.n_best and abs(q - o.modularity) <= (0.0 if g.w is None else 1e-12)


@pytest.mark.parametrize("weights", ["unit", "int", "float"])
@pytest.mark.parametrize("n,entries,hub", [(2, 4, 1), (33, 200, 30), (700, 4000, 90), (2047, 16000, 1500),
                                           (2049, 8000, 300), (4100, 66000, 4000), (8191, 40000, 8100),
                                           (8192, 131000, 5000), (8193, 40000, 100), (3000, 131500, 50)])
def test_limits(n, entries, hub, weights, lv, oracle):
    g = _random(lv, n, entries, hub, weights, n + entries)
    o = oracle.Oracle(g, mode=oracle.SORT, threshold=1e-6)
    o.louvain()
    eng = lv.Engine(0, threshold=1e-6)
    best, q, st = eng.run_graph(g)
    eng.close()
    _check(g, (best, q, st.n_communities), o)


@pytest.mark.parametrize("kw", [dict(mode=0), dict(mode=2, threshold=1e-7), dict(mode=3), dict(fast_first=False),
                                dict(max_levels=2), dict(max_iterations=2), dict(threshold=0.05)])
def test_options_equal_general_path(kw, lv):
    g = _random(lv, 1500, 14000, 400, "unit", 3)
    res = []
    for use_graphs in (False, True):
        eng = lv.Engine(0, use_graphs=use_graphs, **kw)
        best, q, st = eng.run_graph(g)
        res.append((best.tolist(), q, st.levels, st.iterations, st.n_communities, st.active_entries, st.active_vertices))
        eng.close()
    assert res[0] == res[1]


@pytest.mark.parametrize("weights", ["unit", "float"])
def test_batch_of_every_class(weights, lv, oracle):
    """More little graphs than SMs (one CTA each), larger ones on clusters, one for the level loop."""
    batch = importlib.import_module("louvain-fast-move-cuda_b200.batch")
    gs = [_random(lv, 3 + 11 * i, 60 * (i + 1), 2 + i, weights, i) for i in range(170)]
    gs.insert(40, _random(lv, 5000, 60000, 2500, weights, 7))
    gs.insert(90, _random(lv, 12000, 90000, 700, weights, 8))
    offs, row, col, w = batch.pack(gs)
    eng = lv.Engine(0)
    for _ in range(2):
        out, q, k, st = eng.run_batch(offs, row, col, w if weights == "float" else None)
        for i, g in enumerate(gs):
            o = oracle.Oracle(g, mode=oracle.SORT)
            o.louvain()
            _check(g, (out[offs[i]:offs[i + 1]], q[i], k[i]), o)
    eng.close()


def test_bad_input_in_a_batch(lv):
    batch = importlib.import_module("louvain-fast-move-cuda_b200.batch")
    gs = [_random(lv, 40, 200, 5, "unit", i) for i in range(200)]
    offs, row, col, _ = batch.pack(gs)
    eng = lv.Engine(0)
    for at in (0, col.size // 2, col.size - 1):
        bad = col.copy()
        bad[at] = -1
        with pytest.raises(lv.LouvainError) as e:
            eng.run_batch(offs, row, bad)
        assert e.value.status == 2
    out, q, k, _ = eng.run_batch(offs, row, col)
    assert (out >= 0).all()
    eng.close()
