"""Dedispersion of more channels than a grid has rows (65535): taken at native
resolution as before, and the sums are the oracle's."""
import numpy as np
import pytest

import heimdall_multibeam_b200 as H
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nchans", [65536, 70004])
def test_more_channels_than_grid_rows(hdb, oracle_lib, nchans):
    dt, f0, df = 256e-6, 1400.0, -300.0 / nchans
    dms = np.array([0.0, 1.0, 2.5, 9.0], np.float32)
    table = oracle.delay_table(nchans, dt, f0, df)
    nsamps = int(oracle.delays(dms, table).max()) + 131
    fb = np.random.default_rng(1).integers(0, 256, size=(nsamps, nchans), dtype=np.uint8)
    plan = H.DedispPlan(nchans, dt, f0, df)
    plan.set_dm_list(dms)
    np.testing.assert_array_equal(plan.execute(fb), oracle.dedisperse(fb, dms, table))
