"""Device inputs that kernels cannot read where they lie -- at odd addresses, in pinned host memory beside
device arrays -- give what the same arrays give from aligned device memory: they are copied first."""
import importlib
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class At:
    """An array of the C ABI at a raw address (`own` keeps its memory alive)."""
    is_cuda = True

    def __init__(self, own, ptr):
        self.own, self.ptr = own, ptr

    def data_ptr(self):
        return self.ptr


def _put(a, how):
    import torch
    raw = torch.from_numpy(np.frombuffer(np.ascontiguousarray(a).tobytes(), np.uint8).copy())
    if how == "pinned":
        raw = raw.pin_memory()
        return At(raw, raw.data_ptr())
    shift = int(how)  # bytes past an aligned address
    buf = torch.zeros(raw.numel() + 64, dtype=torch.uint8, device="cuda")
    buf[shift:shift + raw.numel()] = raw.cuda()
    torch.cuda.synchronize()
    return At(buf, buf.data_ptr() + shift)


def _graph(lv, weights, n=20_000, m=120_000):
    rng = np.random.default_rng(11)
    u = np.concatenate([np.arange(n), rng.integers(0, n, m)])
    v = np.concatenate([(np.arange(n) + 1) % n, np.minimum(rng.integers(0, n, m), rng.integers(0, n, m))])
    w = None
    if weights == "int":
        w = rng.integers(1, 6, u.size).astype(np.float32)
    elif weights == "float":
        w = (rng.integers(1, 9, u.size) / 4).astype(np.float32)
    return lv.graphs.canonical_from_pairs(u, v, w)


# where row_ptr, col and w lie: 4 is no address for the 8-byte row offsets but one for the others
@pytest.mark.parametrize("row,col,w", [("0", "0", "0"), ("4", "4", "4"), ("0", "1", "0"), ("8", "2", "4"), ("3", "0", "6"),
                                       ("0", "4", "7"), ("0", "pinned", "0"), ("pinned", "0", "pinned"), ("5", "3", "1")])
@pytest.mark.parametrize("weights", ["unit", "int", "float"])
def test_single(row, col, w, weights, lv):
    import torch
    g = _graph(lv, weights)
    eng = lv.Engine(0)
    best, q, st = eng.run_graph(g)
    out = torch.full((g.n,), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    _, q2, st2 = eng.run_csr(g.n, _put(g.row_ptr, row), _put(g.col, col), None if g.w is None else _put(g.w, w), out=out)
    eng.close()
    np.testing.assert_array_equal(out.cpu().numpy(), best)
    assert q2 == q if weights != "float" else abs(q2 - q) < 1e-12
    assert st2.n_communities == st.n_communities


@pytest.mark.parametrize("row,col", [("0", "0"), ("4", "1"), ("pinned", "3")])
def test_batch(row, col, lv):
    import torch
    batch = importlib.import_module("louvain-fast-move-cuda_b200.batch")
    offs, rp, c, _ = batch.pack([_graph(lv, "unit", n, 5 * n) for n in (300, 20_000, 901)])
    eng = lv.Engine(0)
    want, q, k, _ = eng.run_batch(offs, rp, c)
    L, P = eng._L, lv._ptr
    qs, ks, st = np.empty(3), np.empty(3, np.int32), lv.Stats()
    out = np.empty(rp.size - 1, np.int32)
    a, b, o = _put(rp, row), _put(c, col), torch.from_numpy(offs).cuda()
    torch.cuda.synchronize()
    import ctypes
    eng.check(L.lv_run_batch(eng._h, 3, P(o), P(a), P(b), None, lv.MEM_DEVICE, P(out), lv.MEM_HOST,
                             qs.ctypes.data, ks.ctypes.data, ctypes.byref(st)), "lv_run_batch")
    eng.close()
    np.testing.assert_array_equal(out, want)
    np.testing.assert_array_equal(qs, q)
    np.testing.assert_array_equal(ks, k)


SCRIPT = """
import importlib, numpy as np, torch
lv = importlib.import_module("louvain-fast-move-cuda_b200")
n = 3_000_000                                       # (24 MB of row offsets and of columns)
i = torch.arange(n, dtype=torch.int32, device="cuda")
row = torch.arange(n + 1, dtype=torch.int64, device="cuda") * 2
col = torch.stack([(i - 1) % n, (i + 1) % n], 1).reshape(-1).int().contiguous()
out = torch.empty(n, dtype=torch.int32, device="cuda")
torch.cuda.synchronize()
eng = lv.Engine(0)
for _ in range(2):
    eng.run_csr(n, row, col, out=out)
host = eng.run_csr(n, row.cpu().numpy(), col.cpu().numpy())[0]
assert (out.cpu().numpy() == host).all()
print("same")
"""


@pytest.mark.parametrize("conf", ["expandable_segments:True", "backend:cudaMallocAsync"])
def test_allocators(conf):
    """Arrays from allocators that map a segment in pieces, or take it from a stream-ordered pool."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=root, env=dict(os.environ, PYTORCH_CUDA_ALLOC_CONF=conf),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stderr[-2000:]
