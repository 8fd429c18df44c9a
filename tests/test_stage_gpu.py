"""Host copies through the pinned buffers at the sizes where they change hands -- below and above the
smallest staged copy, one byte of a piece more or less, several pieces per thread -- from pageable and
pinned arrays, several calls in a row and several engines at once: bytes in equal bytes out."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ring(lv, n):
    row = np.arange(n + 1, dtype=np.int64) * 2
    i = np.arange(n, dtype=np.int32)
    col = np.stack([(i - 1) % n, (i + 1) % n], 1).reshape(-1).astype(np.int32)
    return lv.graphs.CSRGraph(n=n, row_ptr=row, col=col)


def _round_trip(lv, eng, n):
    g = _ring(lv, n)
    c = eng.community(g)  # uploads row_ptr and col
    row, col, w, k = c.graph()
    c.close()
    np.testing.assert_array_equal(row, g.row_ptr)
    # (rows come back sorted)
    np.testing.assert_array_equal(col.reshape(n, 2), np.sort(g.col.reshape(n, 2), 1))
    assert (k == 2).all() and (w == 1).all()


@pytest.mark.parametrize("n", [32767, 32769, 131071, 131072, 131073, 262145, 1_048_577, 3_000_001])
def test_upload(n, lv):
    eng = lv.Engine(0)
    _round_trip(lv, eng, n)
    _round_trip(lv, eng, n)  # the buffers are in use again
    eng.close()


@pytest.mark.parametrize("n", [40_000, 300_001])
def test_ingest_in_and_out(n, lv):
    g = _ring(lv, n)
    u = np.arange(n)
    text = lv.graphs.edge_list_bytes(u, (u + 1) % n)
    eng = lv.Engine(0)
    for _ in range(2):
        ing = eng.ingest(text)
        c = ing.csr()
        ing.close()
        np.testing.assert_array_equal(c.row_ptr, g.row_ptr)
        np.testing.assert_array_equal(c.col.reshape(n, 2), np.sort(g.col.reshape(n, 2), 1))
    eng.close()


def test_engines_on_threads(lv):
    errs = []

    def work(n):
        try:
            eng = lv.Engine(0)
            for _ in range(3):
                _round_trip(lv, eng, n)
            eng.close()
        except BaseException as e:  # noqa: BLE001 - reported below
            errs.append(e)

    ts = [threading.Thread(target=work, args=(n,)) for n in (500_000, 700_001, 900_003)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errs, errs


def test_loops_of_several_configurations_on_one_engine(lv, graphs, oracle):
    """One engine alternating between configurations of its captured loop (single and batch, with and
    without the heavy-pass walk), more often than it keeps loops."""
    import importlib
    batch = importlib.import_module("louvain-fast-move-cuda_b200.batch")
    gs = [graphs.rmat(15, 8, seed=2), graphs.chung_lu_mean(30000, seed=3), graphs.rmat(17, 24, seed=4)]
    want = []
    for g in gs:
        o = oracle.Oracle(g, mode=oracle.SORT)
        o.louvain()
        want.append((o.best(), o.modularity))
    eng = lv.Engine(0)
    offs, row, col, _ = batch.pack(gs)
    for _ in range(3):
        for g, (best, q) in zip(gs, want):
            r = eng.run_graph(g)
            np.testing.assert_array_equal(r[0], best)
            assert r[1] == q
        out, qs, _, _ = eng.run_batch(offs, row, col)
        for i, (best, q) in enumerate(want):
            np.testing.assert_array_equal(out[offs[i]:offs[i + 1]], best)
            assert qs[i] == q
    eng.close()
