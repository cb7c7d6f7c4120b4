"""Scrunched input rows (adaptive dt) at their edges: lengths around whole
words of outputs for every factor the plan takes, odd lengths, several units,
and a DM list whose factors reach 64; each trial's sums equal the oracle's."""
import numpy as np
import pytest

import heimdall_multibeam_b200 as H
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", [0, 1, 2, 3, 5, 63, 64, 127, 130])
def test_scrunched_sums(hdb, oracle_lib, extra):
    nchans, dt, f0, df = 16, 64e-6, 1200.0, -12.5
    plan = H.DedispPlan(nchans, dt, f0, df)
    dms = np.concatenate([np.linspace(0.0, 20.0, 6), np.geomspace(25.0, 3000.0, 40)])
    plan.set_dm_list(dms)
    plan.enable_adaptive_dt(40.0, 1.15)
    dms = plan.dm_list
    fac = plan.dt_factors
    assert int(fac.max()) >= 16
    nsamps = plan.max_delay + 1024 + extra
    fb = np.random.default_rng(extra).integers(0, 256, size=(nsamps, nchans), dtype=np.uint8)
    got = plan.execute(fb)
    table = oracle.delay_table(nchans, dt, f0, df)
    want = oracle.dedisperse_scrunched(fb, dms, table, fac)
    for d in range(len(dms)):
        np.testing.assert_array_equal(got[d, :len(want[d])], want[d], err_msg=f"trial {d}")
