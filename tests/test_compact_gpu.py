"""The copy of the contracted rows into the next level's graph, at the edges of its chunks of 2,048
entries and of the search for a chunk's rows (33 parts per step): next levels of rows of one entry each
(as many rows in a chunk as it can hold), of a long row over many chunks, and of both in turn. The next
level's edges and weights equal the sums over the partition (whole numbers: bit-exact)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _triangles(count, hub_every):
    """Triangles; with hub_every > 0, each joins the first triangle of its run of hub_every."""
    t = np.arange(count)
    u = np.concatenate([3 * t, 3 * t + 1, 3 * t + 2])
    v = np.concatenate([3 * t + 1, 3 * t + 2, 3 * t])
    if hub_every:
        head = t // hub_every * hub_every
        away = t[t != head]
        u = np.concatenate([u, 3 * away])
        v = np.concatenate([v, 3 * head[away]])
    return u, v


@pytest.mark.parametrize("count,hub_every", [(1, 0), (33, 0), (34, 0), (2047, 0), (2048, 0), (2049, 0), (4097, 0),
                                             (1089 * 33 + 1, 0), (5000, 5000), (6000, 700), (40_000, 3)])
def test_next_level(count, hub_every, lv):
    g = lv.graphs.canonical_from_pairs(*_triangles(count, hub_every))
    eng = lv.Engine(0, threshold=0.0)
    c = eng.community(g)
    c.optimization_step()
    comm, _tot = c.partition()
    row, col, w, k = c.graph()
    src = np.repeat(np.arange(row.size - 1), np.diff(row))
    ids = np.unique(comm)
    new = np.searchsorted(ids, comm)
    want, at = np.unique(new[src].astype(np.int64) * ids.size + new[col], return_inverse=True)
    sums = np.bincount(at, weights=w)
    c.aggregation_run(True)
    row2, col2, w2, _k2 = c.graph()
    eng.close()
    src2 = np.repeat(np.arange(row2.size - 1), np.diff(row2))
    got = src2.astype(np.int64) * ids.size + col2
    order = np.argsort(got)
    assert row2.size - 1 == ids.size
    np.testing.assert_array_equal(got[order], want)
    np.testing.assert_array_equal(np.asarray(w2)[order], sums)
