"""Degree bins so low that every contracted community asks for a global table: below 2^32 slots in all the
result is the oracle's, above the run is refused (and the engine goes on)."""
import numpy as np
import pytest

from test_arena_gpu import _cliques

pytestmark = pytest.mark.gpu
BINS = [1, 1, 2, 2, 4, 4, 4]  # a triangle with two edges to its neighbours: 8 entries, a table of 4,096 slots


@pytest.mark.parametrize("captured", [True, False])
@pytest.mark.parametrize("weights", [False, True])
def test_many_tables(captured, weights, lv, oracle):
    g = _cliques(lv, 100_000, 3, weights)
    o = oracle.Oracle(g, mode=oracle.SORT)
    o.louvain()
    eng = lv.Engine(0, bin_max_degree=BINS, use_graphs=captured)
    best, q, st = eng.run_graph(g)
    eng.close()
    np.testing.assert_array_equal(best, o.best())
    assert abs(q - o.modularity) <= (1e-12 if weights else 0.0) and st.n_communities == o.n_best


@pytest.mark.parametrize("captured", [True, False])
def test_too_many_tables(captured, lv, oracle):
    g = _cliques(lv, 1_100_000, 3)
    o = oracle.Oracle(g, mode=oracle.SORT, nthreads=0)
    o.optimization_run()
    assert np.unique(o.comm()).size * 4096 >= 1 << 32
    small = _cliques(lv, 5_000, 3)
    eng = lv.Engine(0, bin_max_degree=BINS, use_graphs=captured)
    with pytest.raises(lv.LouvainError) as e:
        eng.run_graph(g)
    assert e.value.status == 3  # LV_ERR_RANGE
    want = oracle.Oracle(small, mode=oracle.SORT)
    want.louvain()
    np.testing.assert_array_equal(eng.run_graph(small)[0], want.best())
    eng.close()
