"""A dedispersion call for whose buffers the device has no room fails, and the
plan's next call, which fits, gives the oracle's sums: a buffer that could not
be had counts as empty."""
import os
import sys

import numpy as np
import pytest

import heimdall_multibeam_b200 as H
import oracle

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from device_room import device_room  # noqa: E402

pytestmark = pytest.mark.gpu


# MiB: room for neither copy of the large input (128 MiB each), and for one
@pytest.mark.parametrize("left", [64, 200])
def test_small_call_after_a_failed_large_one(hdb, oracle_lib, left):
    torch = pytest.importorskip("torch")
    nchans, dt, f0, df = 128, 256e-6, 1400.0, -2.0
    dms = np.linspace(0.0, 50.0, 20).astype(np.float32)
    rng = np.random.default_rng(left)
    small = rng.integers(0, 256, size=(4000, nchans), dtype=np.uint8)
    large = np.zeros((1 << 20, nchans), np.uint8)
    plan = H.DedispPlan(nchans, dt, f0, df)
    plan.set_dm_list(dms)
    want = oracle.dedisperse(small, dms, oracle.delay_table(nchans, dt, f0, df))
    np.testing.assert_array_equal(plan.execute(small), want)
    with device_room(torch, left << 20):
        with pytest.raises(RuntimeError, match="Memory allocation failed"):
            plan.execute(large)
        np.testing.assert_array_equal(plan.execute(small), want)
