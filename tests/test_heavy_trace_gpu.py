"""Passes applied by the walk over every row, against the oracle pass by pass: movers, internal weight I
and squared totals S of every record (weights whole or multiples of 1/4, so all sums are exact in
double whatever their order: no tolerance), partition after every pass of the first level. The share of
the level's entries that each pass's movers own is worked out here, and every case has passes on the
side of the walk's limit that it is for."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(lv, n, entries, hubs, seed, weights="unit", near=0):
    """A ring, `hubs` vertices joined to half of all, and random pairs (`near` > 0: up to that far apart)."""
    rng = np.random.default_rng(seed)
    m = entries // 2 - n - hubs * (n // 2)
    at = rng.integers(0, n, m)
    to = (at + rng.integers(1, near + 1, m)) % n if near else rng.integers(0, n, m)
    u = np.concatenate([np.arange(n), np.repeat(rng.integers(0, n, hubs), n // 2), at])
    v = np.concatenate([(np.arange(n) + 1) % n, rng.integers(0, n, hubs * (n // 2)), to])
    w = None
    if weights != "unit":
        w = rng.integers(1, 9, u.size).astype(np.float32) / (4.0 if weights == "float" else 1.0)
        if weights == "float":
            w[0] = 0.25
    return lv.graphs.canonical_from_pairs(u, v, w)


def _rows(tr):
    return [(int(r["level"]), int(r["iteration"]), int(r["n_moved"]), float(r["internal"]), float(r["sum_a2"]))
            for r in tr]


def _shares(eng, g, passes):
    """Per pass of the first level: the entries of its movers over all, and the partition after it."""
    deg = np.diff(g.row_ptr)
    c = eng.community(g)
    before, out = np.arange(g.n), []
    for _ in range(passes):
        c.optimization_step()
        after = c.partition()[0]
        out.append((deg[after != before].sum() / g.E, after))
        before = after
    c.close()
    return out


@pytest.mark.parametrize("n,entries,hubs,near,weights", [
    (60_000, 5_200_000, 0, 0, "unit"), (60_000, 5_200_000, 12, 0, "int"), (200_000, 9_600_000, 3, 60, "float"),
    (400_000, 12_000_000, 1, 30, "float"), (4_000, 6_400_000, 0, 0, "float"),
    (6_100_000, 24_000_000, 0, 9, "unit"), (6_100_000, 24_000_000, 0, 9, "float")])
def test_every_pass(n, entries, hubs, near, weights, lv, oracle):
    g = _graph(lv, n, entries, hubs, n + hubs, weights, near)
    assert g.E >= 1 << 22
    o = oracle.Oracle(g, mode=oracle.SORT, nthreads=0)
    o.louvain()
    want = _rows(o.trace())
    eng = lv.Engine(0)
    c = eng.community(g)
    c.louvain()
    assert _rows(c.trace()) == want
    np.testing.assert_array_equal(c.best(), o.best())
    c.close()
    first = [r for r in want if r[0] == 0]
    step = oracle.Oracle(g, mode=oracle.SORT, nthreads=0)
    shares = _shares(eng, g, min(4, len(first)))
    eng.close()
    for _, part in shares:
        step.optimization_step()
        np.testing.assert_array_equal(part, step.comm())
    walked = [s for s, _ in shares if s > (1 / 6 if n >= 6_000_000 else 1 / 2)]
    assert walked, [s for s, _ in shares]
    if n >= 6_000_000:  # (walked only because of the vertices' number)
        assert any(s <= 1 / 2 for s in walked), walked


def test_batch_float(lv, oracle):
    """Several graphs under one warp's 32 rows, fp32 weights: sums per graph by double atomics."""
    batch = importlib.import_module("louvain-fast-move-cuda_b200.batch")
    gs = [_graph(lv, n, 26 * n, 0, n, "float", 60) for n in (9000, 70_001, 9_001, 40_000, 8_500, 60_000)]
    gs += [_graph(lv, n, 9 * n, 0, n, "float") for n in (8_301, 8_197, 8_231)]
    offs, row, col, w = batch.pack(gs)
    assert col.size >= 1 << 22
    eng = lv.Engine(0)
    out, q, k, _ = eng.run_batch(offs, row, col, w)
    eng.close()
    for i, g in enumerate(gs):
        o = oracle.Oracle(g, mode=oracle.SORT)
        o.louvain()
        np.testing.assert_array_equal(out[offs[i]:offs[i + 1]], o.best())
        assert q[i] == o.modularity and k[i] == o.n_best


@pytest.mark.parametrize("n,entries,hubs,near,weights", [
    (60_000, 5_200_000, 0, 0, "unit"), (200_000, 9_600_000, 6, 60, "int"), (200_000, 9_600_000, 2, 60, "float")])
def test_refined(n, entries, hubs, near, weights, lv, oracle):
    """The walk through the refine view: restricted rows (some empty), rejected proposals among the movers."""
    g = _graph(lv, n, entries, hubs, 7 + hubs, weights, near)
    assert g.E >= 1 << 22
    o = oracle.Oracle(g, mode=oracle.SORT, refine=True, nthreads=0)
    o.louvain()
    for graphs_on in (True, False):
        eng = lv.Engine(0, refine=True, use_graphs=graphs_on)
        c = eng.community(g)
        st = c.louvain()
        assert _rows(c.trace()) == _rows(o.trace())
        np.testing.assert_array_equal(c.best(), o.best())
        assert st.refine_passes == o.refine_passes
        eng.close()
