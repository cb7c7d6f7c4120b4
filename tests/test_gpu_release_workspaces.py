"""The device memory that profiler calls keep for later ones goes back to the
device when the program asks, also while other threads make such calls."""
import threading

import numpy as np
import pytest

import heimdall_multibeam_b200 as H

pytestmark = pytest.mark.gpu


def test_profiler_memory_is_given_back(hdb):
    torch = pytest.importorskip("torch")
    nsamps, nchans = 1 << 17, 256
    fb = np.random.default_rng(2).integers(0, 256, size=(nsamps, nchans), dtype=np.uint8)
    dms = np.linspace(0.0, 300.0, 60, dtype=np.float32)
    reqs = [(20000 + 3000 * k, k % 6, 5 + 4 * k) for k in range(12)]

    def profile():
        return H.profile_candidates(fb, 64e-6, 1500.0, -400.0 / nchans, dms, reqs)

    want = profile()
    H.release_workspaces()
    free = torch.cuda.mem_get_info()[0]
    profile()
    assert torch.cuda.mem_get_info()[0] < free - nsamps * nchans // 2
    H.release_workspaces()
    assert torch.cuda.mem_get_info()[0] >= free - (8 << 20)
    bad = []

    def calls():
        for _ in range(6):
            for a, b in zip(profile(), want):
                bad.extend(k for k in b if not np.array_equal(a[k], b[k], equal_nan=True))

    threads = [threading.Thread(target=calls) for _ in range(3)]
    for t in threads:
        t.start()
    while any(t.is_alive() for t in threads):
        H.release_workspaces()
    for t in threads:
        t.join()
    assert not bad
    H.release_workspaces()
    assert torch.cuda.mem_get_info()[0] >= free - (8 << 20)
