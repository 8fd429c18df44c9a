"""Contraction kernels at the edges of their shapes: communities of 1 to 33 entries (all pairs), of one
member or of many one-entry members, of 33 to a few thousand entries (warp, block), and large ones
(global tables), under the built-in bins and configured ones on both sides of the pair limit. The
contracted graph -- destinations, weights, row sums -- equals the dense sum over the partition (whole-number
weights: bit-exact; fp32 weights that are multiples of 1/4: sums exact, so equal too)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(lv, weights, seed):
    """Cliques, stars and paths of many sizes, joined by random edges."""
    rng = np.random.default_rng(seed)
    us, vs, base = [], [], 0
    for k in (2, 3, 4, 5, 6, 7, 9, 12, 30, 70):          # cliques
        for _ in range(6):
            i, j = np.triu_indices(k, 1)
            us.append(base + i)
            vs.append(base + j)
            base += k
    for k in (2, 3, 4, 15, 16, 31, 32, 33, 500, 5000):    # stars: many one-entry members
        us.append(np.full(k, base))
        vs.append(base + 1 + np.arange(k))
        base += k + 1
    n = base
    us.append(rng.integers(0, n, 600))
    vs.append(rng.integers(0, n, 600))
    u, v = np.concatenate(us), np.concatenate(vs)
    w = None
    if weights != "unit":
        w = rng.integers(1, 9, u.size).astype(np.float32) / (4.0 if weights == "float" else 1.0)
    return lv.graphs.canonical_from_pairs(u, v, w)


@pytest.mark.parametrize("weights", ["unit", "int", "float"])
@pytest.mark.parametrize("bins", [None, (8, 16, 32, 64, 128, 512, 2048), (2, 6, 31, 33, 40, 300, 1000), (4, 8, 40, 48, 128, 256, 512)])
def test_levels(bins, weights, lv):
    g = _graph(lv, weights, 3)
    eng = lv.Engine(0, threshold=0.0, bin_max_degree=bins)
    c = eng.community(g)
    for _ in range(2):
        c.optimization_run()
        comm, _tot = c.partition()
        row, col, w, k = c.graph()
        src = np.repeat(np.arange(row.size - 1), np.diff(row))
        ids = np.unique(comm)
        new = np.searchsorted(ids, comm)
        want = np.zeros((ids.size, ids.size))
        np.add.at(want, (new[src], new[col]), w)
        c.aggregation_run(True)
        row2, col2, w2, k2 = c.graph()
        got = np.zeros_like(want)
        src2 = np.repeat(np.arange(row2.size - 1), np.diff(row2))
        np.add.at(got, (src2, col2), w2)
        assert row2.size - 1 == ids.size and row2[-1] == np.count_nonzero(want)  # one entry per pair
        np.testing.assert_array_equal(got, want)
        np.testing.assert_array_equal(k2, want.sum(1))
        break_if = row2.size - 1 < 3
        if break_if:
            break
    eng.close()


@pytest.mark.parametrize("weights", ["unit", "int", "float"])
def test_whole_run(weights, lv, oracle):
    g = _graph(lv, weights, 9)
    o = oracle.Oracle(g, mode=oracle.SORT)
    o.louvain()
    for bins in (None, (4, 8, 16, 32, 64, 128, 300)):
        eng = lv.Engine(0, bin_max_degree=bins)
        best, q, st = eng.run_graph(g)
        eng.close()
        np.testing.assert_array_equal(best, o.best())
        assert st.n_communities == o.n_best and abs(q - o.modularity) <= 1e-12
