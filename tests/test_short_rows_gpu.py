"""Rows at the edges of the short-row gain kernel's shapes (4 T entries for T = 1, 2, 4, 8 lanes, and
one entry more or less): final partition, community count and modularity against the oracle.
Exact for whole-number weights and for fp32 weights that are multiples of 1/4 (every sum is exact
in double); 1e-12 on Q covers the order of the squared totals' sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(lv, degrees, copies, weights, seed):
    """Disjoint circulant graphs, one per degree, tied together by a few long edges."""
    rng = np.random.default_rng(seed)
    us, vs, base = [], [], 0
    for d in degrees:
        n = 2 * d + 3
        for _ in range(copies):
            i = np.arange(n)
            for k in range(1, d // 2 + 1):
                us.append(base + i)
                vs.append(base + (i + k) % n)
            if d % 2:  # odd degree: a perfect matching between two halves, one vertex short
                h = n // 2
                us.append(base + i[:h])
                vs.append(base + h + i[:h])
            base += n
    us.append(rng.integers(0, base, 40))
    vs.append(rng.integers(0, base, 40))
    u, v = np.concatenate(us), np.concatenate(vs)
    w = None
    if weights == "int":
        w = rng.integers(1, 8, u.size).astype(np.float32)
    elif weights == "float":
        w = (rng.integers(1, 8, u.size) / 4.0).astype(np.float32)
    return lv.graphs.canonical_from_pairs(u, v, w)


@pytest.mark.parametrize("mode", ["SORT", "HASH"])
@pytest.mark.parametrize("weights", ["unit", "int", "float"])
@pytest.mark.parametrize("degrees", [(1, 2, 3, 4, 5), (7, 8, 9, 15), (16, 17, 31), (32, 33, 4, 1)])
def test_edges(degrees, weights, mode, lv, oracle):
    g = _graph(lv, degrees, 7, weights, sum(degrees))
    o = oracle.Oracle(g, mode=getattr(oracle, mode))
    o.louvain()
    eng = lv.Engine(0, mode=lv.MODE[mode])
    best, q, st = eng.run_graph(g)
    eng.close()
    np.testing.assert_array_equal(best, o.best())
    assert st.n_communities == o.n_best and abs(q - o.modularity) <= 1e-12


@pytest.mark.parametrize("bins", [(1, 2, 4, 8, 32, 64, 256), (5, 9, 17, 33, 64, 128, 512), (4, 12, 16, 48, 64, 96, 128)])
def test_bin_limits(bins, lv, oracle):
    """Configured limits below, at and above what the kernel holds (above: the table kernel)."""
    g = _graph(lv, (1, 3, 5, 9, 17, 33, 47), 3, "unit", 5)
    o = oracle.Oracle(g, mode=oracle.SORT)
    o.louvain()
    eng = lv.Engine(0, bin_max_degree=bins)
    best, q, st = eng.run_graph(g)
    eng.close()
    np.testing.assert_array_equal(best, o.best())
    assert st.n_communities == o.n_best and abs(q - o.modularity) <= 1e-12
