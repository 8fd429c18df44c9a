"""Level-0 input kernels at the edges of their 32-vertex ranges: row sums, total weight and
self-loop weight against plain sums (exact: whole numbers, or fp32 weights that are multiples of
1/4), and the column check in every path."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(lv, n, pairs, weighted, seed=0):
    rng = np.random.default_rng(seed)
    rows = [[] for _ in range(n)]
    for u, v in pairs:
        w = float(rng.integers(1, 9)) / 4.0 if weighted else 1.0
        rows[u].append((v, w))
        rows[v].append((u, w))  # a self-loop is stored twice, as the edge-list loader does
    row = np.zeros(n + 1, np.int64)
    row[1:] = np.cumsum([len(r) for r in rows])
    col = np.array([v for r in rows for v, _ in r], np.int32)
    w = np.array([x for r in rows for _, x in r], np.float32)
    return lv.graphs.CSRGraph(n=n, row_ptr=row, col=col, w=w if weighted else None)


def _shape(name):
    if name.startswith("ring"):  # loops at the first and last vertex of the ranges
        n = int(name[4:])
        return n, [(i, (i + 1) % n) for i in range(n)] + [(i, i) for i in (0, 31, 32, n - 1) if i < n]
    n = int(name[3:])            # a hub row inside one range, loops on the hub and behind it
    return n, [(5, i) for i in range(n) if i != 5] + [(5, 5), (33, 33), (n - 1, n - 1)]


SHAPES = ["ring31", "ring32", "ring33", "ring65", "hub513", "hub1025", "hub8160", "hub8200", "hub20000"]


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("name", SHAPES)
def test_sums(name, weighted, lv):
    n, pairs = _shape(name)
    g = _csr(lv, n, pairs, weighted)
    x = g.weights_or_ones.astype(np.float64)
    src = g.src()
    eng = lv.Engine(0, weight_mode=lv.WEIGHTS_FLOAT if weighted else lv.WEIGHTS_AUTO)
    c = eng.community(g)
    info = c.info()
    row, col, w, k = c.graph()
    np.testing.assert_array_equal(row, g.row_ptr)
    np.testing.assert_array_equal(k, np.bincount(src, weights=x, minlength=n))
    np.testing.assert_array_equal(np.bincount(np.repeat(np.arange(n), np.diff(row)), weights=w, minlength=n), k)
    assert info.total_weight == x.sum() / 2 and info.internal == x[src == g.col].sum()
    eng.close()


@pytest.mark.parametrize("name,at", [("ring33", 5), ("hub8160", 4000), ("hub20000", 19000), ("hub20000", 39995)])
@pytest.mark.parametrize("weighted", [False, True])
def test_column_out_of_range(name, at, weighted, lv):
    n, pairs = _shape(name)
    g = _csr(lv, n, pairs, weighted)
    g.col[at] = n
    eng = lv.Engine(0)
    with pytest.raises(lv.LouvainError) as e:
        eng.run_graph(g)
    assert e.value.status == 2
    eng.close()


def test_ranges_spanning_graphs(lv, oracle):
    """Tiny graphs (several per 32-vertex range) beside one whose hub row spans pieces."""
    import importlib
    batch = importlib.import_module("louvain-fast-move-cuda_b200.batch")
    gs = [_csr(lv, n, [(i, (i + 1) % n) for i in range(n)] + [(n - 1, n - 1), (0, 0)], False) for n in (3, 4, 7, 13, 30)]
    gs.insert(2, _csr(lv, *_shape("hub9000"), False))
    offs, row, col, _ = batch.pack(gs)
    eng = lv.Engine(0)
    out, q, k, _ = eng.run_batch(offs, row, col)
    for i, g in enumerate(gs):
        o = oracle.Oracle(g, mode=oracle.SORT)
        o.louvain()
        np.testing.assert_array_equal(out[offs[i]:offs[i + 1]], o.best())
        assert q[i] == o.modularity and k[i] == o.n_best
    bad = col.copy()
    bad[0] = offs[1]  # inside the batch, outside its own graph
    with pytest.raises(lv.LouvainError):
        eng.run_batch(offs, row, bad)
    eng.close()
