"""A served request takes no more device memory than its server may use: the arena that a run likes to have
ahead of its need is taken only where the budget has room for it."""
import numpy as np
import pytest

from test_arena_gpu import MB, _cliques

pytestmark = pytest.mark.gpu


def _drop(lv, g, small, budget, slots):
    """Bytes of device memory that serving `g` takes on a server already running."""
    import torch
    eng = lv.Engine(0)
    srv = lv.Server(eng, budget, slots=slots)
    def serve(x):
        i = srv.submit(x)
        srv.drain()
        return srv.poll(i)
    for _ in range(2 * slots):  # kernels loaded, loops captured
        serve(small)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    res = serve(g)
    torch.cuda.synchronize()
    drop = before - torch.cuda.mem_get_info()[0]
    srv.close()
    eng.close()
    return drop, res


def test_memory_stays_in_the_budget(lv):
    g = _cliques(lv, 16_000, 40)          # 25 M entries, no table of any size needed
    small = _cliques(lv, 700, 40)
    est = g.E * 16 + g.n * 124            # what it is admitted for
    eng = lv.Engine(0)
    want = eng.run_graph(g)[:2]
    eng.close()
    # a budget a quarter above the estimate, and one with room for everything the run would like
    tight, roomy = est + est // 4, 64 << 30
    drop, res = _drop(lv, g, small, tight, 1)
    np.testing.assert_array_equal(res[0], want[0])
    assert res[1] == want[1]
    assert drop <= tight, (drop // MB, tight // MB)
    drop2, res = _drop(lv, g, small, roomy, 1)
    np.testing.assert_array_equal(res[0], want[0])
    assert drop2 > drop + 300 * MB        # (there the arena is taken: 48 M slots of 8 bytes)


def test_share_of_a_slot(lv):
    """With several slots the arena ahead of need stays within the slot's share of the budget."""
    g = _cliques(lv, 16_000, 40)
    est = g.E * 16 + g.n * 124
    drop, _ = _drop(lv, g, _cliques(lv, 700, 40), 4 * est, 4)  # the estimate alone is the share
    assert drop <= est + est // 4, (drop // MB, est // MB)
