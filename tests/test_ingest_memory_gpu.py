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


def test_kept(lv):
    """After it, the engine keeps no more than a gigabyte, whatever it was; and a small ingest's buffers, which
    the next one takes again."""
    small, large = _text(lv, 200_000, 1_000_000), _text(lv, 1_000_000, 45_000_000)
    eng = _warm(lv)
    start = _free()
    eng.ingest(small).close()
    one = start - _free()
    eng.ingest(small).close()
    assert start - _free() == one
    ing = eng.ingest(large)
    want = ing.csr()
    ing.close()
    assert start - _free() <= 1024 * MB + 64 * MB, (start - _free()) // MB
    again = eng.ingest(large)
    got = again.csr()
    np.testing.assert_array_equal(got.row_ptr, want.row_ptr)
    np.testing.assert_array_equal(got.col, want.col)
    again.close()
    assert start - _free() <= 1024 * MB + 64 * MB, (start - _free()) // MB
    eng.close()
    assert start - _free() <= 64 * MB
