"""The module functions called by several host threads at once, as one thread per body or per stream would."""
import threading

import numpy as np
import pytest

import oracle as O
import vpd

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_neighbor_lists_built_by_four_threads():
    """Horizons of 2, 3, 4.015 and 5 spacings: 216 to 3,375 candidates around a cell, so every thread's search
    stages another amount of shared memory."""
    pos = np.stack(np.meshgrid(np.arange(24), np.arange(13), np.arange(12), indexing="ij"), -1).reshape(-1, 3) * 1.0
    want = {}
    for horizon in (2.0, 3.0, 4.015, 5.0):
        row_ptr, col = O.neighbor_list(np.ascontiguousarray(pos), horizon)
        want[horizon] = torch.as_tensor(row_ptr).cuda(), torch.as_tensor(col[:row_ptr[-1]]).cuda()
    x = torch.as_tensor(pos).cuda()
    torch.cuda.synchronize()
    failures = []
    start = threading.Barrier(len(want))

    def build(horizon):
        stream = torch.cuda.Stream()
        start.wait()
        try:
            with torch.cuda.stream(stream):
                for _ in range(300):
                    row_ptr, col = vpd.build_neighbor_list(x, horizon)
                    assert torch.equal(row_ptr, want[horizon][0]) and torch.equal(col, want[horizon][1])
        except Exception as e:  # reported by the main thread
            failures.append((horizon, repr(e)))

    threads = [threading.Thread(target=build, args=(h,)) for h in want]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures
