"""Device memory of an ingest: what it takes while it runs, and what the engine keeps of it afterwards."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _text(lv, n, pairs):
    rng = np.random.default_rng(1)
    u = np.concatenate([np.arange(n), rng.integers(0, n, pairs - n)])
    v = np.concatenate([(np.arange(n) + 1) % n, rng.integers(0, n, pairs - n)])
    return np.frombuffer(lv.graphs.edge_list_bytes(u, v), np.uint8)


def _warm(lv):
    import torch
    torch.cuda.init()
    eng = lv.Engine(0)
    eng.ingest(_text(lv, 1000, 5000)).close()  # kernels loaded
    return eng


def test_taken(lv):
    """The text, the positions (8 bytes a token) and values (4) of its tokens, the rows in the positions'
    block, the columns in the values', and 40 bytes per vertex."""
    n, pairs = 1_000_000, 20_000_000
    text = _text(lv, n, pairs)
    eng = _warm(lv)
    before = _free()
    ing = eng.ingest(text)
    taken = before - _free()
    assert ing.n_nodes == n
    ing.close()
    eng.close()
    assert taken <= text.size + 2 * pairs * 12 + n * 40 + 64 * MB, taken // MB
