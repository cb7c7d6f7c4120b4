"""Dedispersion over four-sample words at the sizes where it can go wrong:
output lengths around the rounding of the quarter length (16 words) and of a
tile's words, channel counts around the runs of 256 channels between two
flushes of the packed sums (all bytes 255, the largest sums), and trials so far
apart that only the tiles of two trials or of one fit shared memory.  The sums
are whole numbers, so they equal the oracle's exactly."""
import numpy as np
import pytest

import heimdall_multibeam_b200 as H
import oracle

pytestmark = pytest.mark.gpu


def _check(nchans, nsamps, dt, f0, df, dms, full=False, killmask=None):
    rng = np.random.default_rng(nchans * 1000003 + nsamps)
    fb = np.full((nsamps, nchans), 255, np.uint8) if full else \
        rng.integers(0, 256, size=(nsamps, nchans), dtype=np.uint8)
    plan = H.DedispPlan(nchans, dt, f0, df)
    dms = np.asarray(dms, np.float32)
    plan.set_dm_list(dms)
    if killmask is not None:
        plan.set_killmask(killmask)
    table = oracle.delay_table(nchans, dt, f0, df)
    np.testing.assert_array_equal(plan.execute(fb), oracle.dedisperse(fb, dms, table, killmask))


@pytest.mark.parametrize("nout", [1, 3, 15, 16, 17, 63, 64, 65, 1279, 1280, 1281, 5120, 5121])
def test_output_lengths(hdb, oracle_lib, nout):
    dms = [0.0, 5.0, 40.0, 41.0, 90.0, 150.0, 151.0, 152.0, 200.0]
    table = oracle.delay_table(16, 256e-6, 1400.0, -6.0)
    md = int(oracle.delays(np.asarray(dms, np.float32), table).max())
    _check(16, md + nout, 256e-6, 1400.0, -6.0, dms)


@pytest.mark.parametrize("nchans", [4, 252, 256, 260, 512, 516, 772])
def test_channel_runs(hdb, oracle_lib, nchans):
    dms = np.linspace(0.0, 60.0, 11)
    _check(nchans, 3000, 256e-6, 1400.0, -200.0 / nchans, dms, full=True)
    km = np.ones(nchans, np.int32)
    km[1::7] = 0
    _check(nchans, 2999, 256e-6, 1400.0, -200.0 / nchans, dms, killmask=km)


@pytest.mark.parametrize("step", [60.0, 200.0, 380.0])
def test_trials_far_apart(hdb, oracle_lib, step):
    """8-trial spans of about 10, 33 and 63 thousand samples: the last two fit
    no block of eight trials."""
    nchans, df = 32, -12.5
    dms = np.arange(9) * step
    table = oracle.delay_table(nchans, 64e-6, 1520.0, df)
    md = int(oracle.delays(dms.astype(np.float32), table).max())
    _check(nchans, md + 9001, 64e-6, 1520.0, df, dms)


def test_trials_too_far_apart_are_refused(hdb):
    plan = H.DedispPlan(32, 64e-6, 1520.0, -12.5)
    plan.set_dm_list(np.arange(40) * 450.0)
    with pytest.raises(RuntimeError, match="exceeds internal limit"):
        plan.execute(np.zeros((450000, 32), np.uint8))
