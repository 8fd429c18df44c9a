"""lv_ingest_copy_csr: ordered behind the work queued for its destination, and not held up by another
call of the same context."""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ring(lv, eng, n):
    u = np.arange(n)
    ing = eng.ingest(lv.graphs.edge_list_bytes(u, (u + 1) % n))
    return ing, ing.csr()


@pytest.mark.parametrize("n", [1000, 400_001])  # (in host memory: below and above the smallest staged copy)
@pytest.mark.parametrize("where", ["device", "pinned"])
def test_order(n, where, lv):
    import torch
    eng = lv.Engine(0)
    ing, want = _ring(lv, eng, n)
    row, col = torch.empty(n + 1, dtype=torch.int64), torch.empty(2 * n, dtype=torch.int32)
    minus = torch.full((2 * n,), -1, dtype=torch.int64, device="cuda")
    if where == "device":
        row, col = row.cuda(), col.cuda()
    else:
        row, col = row.pin_memory(), col.pin_memory()
    torch.cuda.synchronize()
    # the default stream is busy for a tenth of a second, then overwrites the destinations
    torch.cuda._sleep(200_000_000)
    row.copy_(minus[: n + 1], non_blocking=True)
    col.copy_(minus, non_blocking=True)
    eng.check(eng._L.lv_ingest_copy_csr(ing._h, row.data_ptr(), col.data_ptr(),
                                        lv.MEM_DEVICE if where == "device" else lv.MEM_HOST), "copy")
    torch.cuda.synchronize()
    np.testing.assert_array_equal(row.cpu().numpy(), want.row_ptr)
    np.testing.assert_array_equal(col.cpu().numpy(), want.col)
    ing.close()
    eng.close()


@pytest.mark.parametrize("where", ["device", "host"])
def test_beside_another_call(where, lv, graphs):
    """Copies while another thread's calls keep the context busy: right, and most of them done before the
    call they met has ended."""
    import torch
    eng = lv.Engine(0)
    n = 1000
    ing, want = _ring(lv, eng, n)
    big = graphs.rmat(18, 16, seed=1)
    eng.run_graph(big)
    stop, spans = threading.Event(), []

    def busy():
        while not stop.is_set():
            t = time.perf_counter()
            eng.run_graph(big)
            spans.append((t, time.perf_counter()))

    th = threading.Thread(target=busy)
    th.start()
    done = []
    time.sleep(0.05)
    for _ in range(40):
        row, col = torch.empty(n + 1, dtype=torch.int64), torch.empty(2 * n, dtype=torch.int32)
        if where == "device":
            row, col = row.cuda(), col.cuda()
        t = time.perf_counter()
        eng.check(eng._L.lv_ingest_copy_csr(ing._h, row.data_ptr(), col.data_ptr(),
                                            lv.MEM_DEVICE if where == "device" else lv.MEM_HOST), "copy")
        done.append((t, time.perf_counter()))
        np.testing.assert_array_equal(row.cpu().numpy(), want.row_ptr)
        np.testing.assert_array_equal(col.cpu().numpy(), want.col)
        time.sleep(0.003)
    stop.set()
    th.join()
    met = [(a, b) for a, b in done if any(s < a < e for s, e in spans)]
    inside = [1 for a, b in met if any(s < a and b < e for s, e in spans)]
    ing.close()
    eng.close()
    assert len(met) >= 20 and 2 * len(inside) > len(met), (len(met), len(inside))
