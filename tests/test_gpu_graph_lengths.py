"""Single gulps whose length varies on one pipeline: ten lengths in turn, more
than the pipeline captures at once.  Every gulp gives what the host-sized path
gives, lengths that come back often enough are replayed in the end, and a cycle
takes no longer than without graphs (a capture costs several such gulps, so a
graph that is captured again on each call shows)."""
import time

import numpy as np
import pytest

import heimdall_multibeam_b200 as H
from heimdall_multibeam_b200 import synth

pytestmark = pytest.mark.gpu

LENGTHS = [8192 + 411 * k for k in range(10)]


@pytest.mark.parametrize("device", [False, True])
def test_cycled_lengths(hdb, device):
    torch = pytest.importorskip("torch")
    p = H.default_params(nchans=64, dt=655.36e-6, f0=851.0, df=-0.390625, dm_max=600.0,
                         boxcar_max=256, output_dir=None)
    fbs = [synth.make_beam(n, 64, 655.36e-6, 851.0, -0.390625,
                           [synth.Pulse(2000.0 + 50 * k, 200.0, 5e-3, 30.0)], seed=k).data
           for k, n in enumerate(LENGTHS)]
    d = [torch.from_numpy(fb).cuda() for fb in fbs]

    def gulp(pl, k):
        if device:
            return pl.execute_device(d[k].data_ptr(), LENGTHS[k])
        return pl.execute(fbs[k], raise_on_error=False)

    def result(pl, r):
        g = pl.giants()
        return r, H.cand_lines(pl.candidates()), {k: np.asarray(v).tolist() for k, v in g.items()}

    with H.Pipeline(p, cleaning=False) as on, H.Pipeline(p, cleaning=False) as off:
        off.set_graphs(False)
        want = [result(off, gulp(off, k)) for k in range(10)]
        assert sum(len(w[1]) for w in want) >= 10
        cycles = {on: [], off: []}
        for c in range(50):
            for pl in (on, off):
                torch.cuda.synchronize()
                t = time.perf_counter()
                for k in range(10):
                    gulp(pl, k)
                cycles[pl].append(time.perf_counter() - t)
            if c in (0, 1, 30, 40, 49):
                for k in range(10):
                    assert result(on, gulp(on, k)) == want[k], (c, k)
        assert on.graph_replays() >= 10 and off.graph_replays() == 0
    # the first cycle allocates; of the others one at most captures
    a, b = sorted(cycles[on][1:]), sorted(cycles[off][1:])
    assert a[len(a) // 2] <= 1.25 * b[len(b) // 2], (a, b)
    assert sum(a) <= 2.5 * sum(b), (a, b)
