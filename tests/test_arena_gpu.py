"""The hash-table arena that a run takes ahead of its need: only from memory that is to spare."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _cliques(lv, count, size, w=False):
    """`count` cliques, one edge from each to the next (no community of more than 4,096 entries at level 0)."""
    at = np.arange(count)[:, None] * size
    a, b = np.triu_indices(size, 1)
    u = np.concatenate([(at + a).ravel(), at.ravel()])
    v = np.concatenate([(at + b).ravel(), (np.roll(at, -1, 0) + 1).ravel()])
    g = lv.graphs.canonical_from_pairs(u, v)
    return lv.graphs.CSRGraph(n=g.n, row_ptr=g.row_ptr, col=g.col, w=np.full(g.E, 0.75, np.float32) if w else None)


def test_no_other_blocks_given_up(lv):
    """A run that finds too little memory for the arena it would like keeps the pool's other blocks in place
    and takes what it needs: its result is the same, and the device has no more free memory after it."""
    import torch
    eng = lv.Engine(0, weight_mode=lv.WEIGHTS_FLOAT)
    plain = _cliques(lv, 16_000, 40)
    weighted = _cliques(lv, 16_000, 40, True)
    wide = _cliques(lv, 1_000_000, 3)  # other block sizes than the runs on `plain` and `weighted`
    torch.cuda.init()
    want = eng.run_graph(weighted)[:2]   # loads and captures what that run needs
    eng.close()
    eng = lv.Engine(0, weight_mode=lv.WEIGHTS_FLOAT)
    eng.run_graph(plain)  # whole-number sums: 8 bytes per slot, 12 for `weighted`
    eng.run_graph(wide)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    hold = torch.empty(free - 220 * MB, dtype=torch.uint8, device="cuda")
    before = torch.cuda.mem_get_info()[0]
    got = eng.run_graph(weighted)[:2]
    after = torch.cuda.mem_get_info()[0]
    del hold
    torch.cuda.empty_cache()
    eng.close()
    np.testing.assert_array_equal(got[0], want[0])
    assert abs(got[1] - want[1]) <= 1e-12
    assert after <= before, (before // MB, after // MB)
