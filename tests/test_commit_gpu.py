"""Per-graph squared totals of a packed batch where graphs begin and end inside the commit kernel's
spans and warps (512 and 32 vertices): modularity and partition per graph equal to the oracle's
(integer weights, exact). The general path is forced by a caller's degree bin."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(511, 1, 512, 2, 513), (32, 31, 33, 480, 1024), (5, 3, 2000, 7, 40, 1500, 20)])
@pytest.mark.parametrize("mode", ["SORT", "HASH"])
def test_spans(sizes, mode, lv, oracle):
    batch = importlib.import_module("louvain-fast-move-cuda_b200.batch")
    gs = []
    for i, n in enumerate(sizes):
        rng = np.random.default_rng(n + i)
        ring = np.arange(n)
        u = np.concatenate([ring, rng.integers(0, n, 3 * n)])
        v = np.concatenate([(ring + 1) % n, rng.integers(0, n, 3 * n)])
        if n > 2:
            gs.append(lv.graphs.canonical_from_pairs(u, v))
        else:  # one or two vertices: self-loops, stored twice
            row = np.arange(n + 1, dtype=np.int64) * 2
            gs.append(lv.graphs.CSRGraph(n=n, row_ptr=row, col=np.repeat(np.arange(n, dtype=np.int32), 2)))
    offs, row, col, _ = batch.pack(gs)
    eng = lv.Engine(0, mode=lv.MODE[mode], bin_max_degree=[3, 8, 16, 32, 128, 512, 4096])
    out, q, k, _ = eng.run_batch(offs, row, col)
    eng.close()
    for i, g in enumerate(gs):
        o = oracle.Oracle(g, mode=getattr(oracle, mode))
        o.louvain()
        np.testing.assert_array_equal(out[offs[i]:offs[i + 1]], o.best())
        assert q[i] == o.modularity and k[i] == o.n_best
