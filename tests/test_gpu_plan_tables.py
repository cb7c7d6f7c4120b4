"""What a dedispersion plan keeps on the device beside its delays: the delay
ranges of blocks of 8, 16 and 32 trials (7/16 of the delay table's bytes), not
those of one and of two trials, which only plans with trials far apart use."""
import numpy as np
import pytest

import heimdall_multibeam_b200 as H
import oracle

pytestmark = pytest.mark.gpu


def test_device_memory_of_a_plan(hdb, oracle_lib):
    torch = pytest.importorskip("torch")
    nchans, trials, dt, f0, df = 1024, 4000, 256e-6, 1400.0, -0.25
    dms = np.linspace(0.0, 100.0, trials).astype(np.float32)
    table = oracle.delay_table(nchans, dt, f0, df)
    nsamps = int(oracle.delays(dms, table).max()) + 61
    fb = np.random.default_rng(3).integers(0, 256, size=(nsamps, nchans), dtype=np.uint8)
    want = oracle.dedisperse(fb, dms, table)

    def used(n):
        plan = H.DedispPlan(nchans, dt, f0, df)
        plan.set_dm_list(dms[:n])
        before = torch.cuda.mem_get_info()[0]
        out = plan.execute(fb)
        np.testing.assert_array_equal(out[:, :61], want[:n, :61])
        return before - torch.cuda.mem_get_info()[0]

    few = used(8)  # (also loads the kernels; its input buffers are as large)
    few = used(8)
    delays = 4 * trials * nchans
    out_bytes = 4 * trials * (nsamps + 3)
    assert used(trials) - few <= 1.5 * delays + out_bytes + (8 << 20)


@pytest.mark.parametrize("trials", [1, 2, 7, 8, 9, 31, 33, 64, 65])
@pytest.mark.parametrize("step", [0.7, 3.0, 380.0])
def test_ranges_of_trial_counts(hdb, oracle_lib, trials, step):
    """Last blocks of every size, for tiles of many trials and of few."""
    nchans, dt, f0, df = 16, 64e-6, 1520.0, -25.0
    if step > 100 and trials > 9:
        trials = 9 + trials % 2
    dms = (np.arange(trials) * step).astype(np.float32)
    table = oracle.delay_table(nchans, dt, f0, df)
    nsamps = int(oracle.delays(dms, table).max()) + 2003
    fb = np.random.default_rng(trials).integers(0, 256, size=(nsamps, nchans), dtype=np.uint8)
    plan = H.DedispPlan(nchans, dt, f0, df)
    plan.set_dm_list(dms)
    np.testing.assert_array_equal(plan.execute(fb), oracle.dedisperse(fb, dms, table))
