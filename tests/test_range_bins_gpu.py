"""Contraction by ranges under degree bins that let bin 7 begin below the smallest community it takes:
thousands of communities on both sides of that size, against the oracle (whole-number sums: exact)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cliques(lv, sizes):
    """Cliques of the given sizes, one edge from each to the next."""
    first = np.concatenate([[0], np.cumsum(sizes)])
    us, vs = [first[:-1]], [np.roll(first[:-1], -1) + 1]
    for s in np.unique(sizes):
        a, b = np.triu_indices(s, 1)
        at = first[:-1][sizes == s][:, None]
        us.append((at + a).ravel())
        vs.append((at + b).ravel())
    return lv.graphs.canonical_from_pairs(np.concatenate(us), np.concatenate(vs))


@pytest.mark.parametrize("top", [512, 2047])
def test_low_bins(top, lv, oracle):
    # 33 vertices: 1,058 entries; 50 vertices: 2,452 (with the two edges to the neighbours)
    g = _cliques(lv, np.random.default_rng(3).permutation(np.repeat([33, 50], [8000, 3500])))
    assert g.E >= 1 << 24
    o = oracle.Oracle(g, mode=oracle.SORT)
    o.louvain()
    eng = lv.Engine(0, bin_max_degree=[4, 8, 16, 32, 128, 512, top])
    best, q, st = eng.run_graph(g)
    eng.close()
    np.testing.assert_array_equal(best, o.best())
    assert q == o.modularity and st.n_communities == o.n_best
