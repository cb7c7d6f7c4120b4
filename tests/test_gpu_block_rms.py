"""Block RMS of series whose median trees have two to five levels in the first
pass, with groups that begin at each alignment, more groups than one block
takes, few and many widths, and non-finite series: candidates and giants equal
the oracle's bit for bit."""
import os
import sys

import numpy as np
import pytest

import heimdall_multibeam_b200 as H
from heimdall_multibeam_b200 import synth

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from test_gpu_parity import _compare  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("boxcar_max,n", [
    (8, 60), (8, 140), (16, 700), (32, 3300), (8, 3 * 3125 + 40), (2048, 11 * 3125 + 2100),
    (256, 27 * 3125 + 300)])
def test_levels_and_groups(hdb, oracle_lib, boxcar_max, n):
    w = synth.Workload("b", 64, 128e-6, 1400.0, -4.0, 0, 1, 0.0, 20.0, boxcar_max, False, "")
    n += int(synth.max_delay_samples(w.dm_max, w.nchans, w.dt, w.f0, w.df)) + 1
    b = synth.make_beam(n, w.nchans, w.dt, w.f0, w.df,
                        [synth.Pulse(n * 0.3, 10.0, 2e-4, 60.0),
                         synth.Pulse(n * 0.6, 15.0, boxcar_max * w.dt / 4, 60.0)], seed=n)
    w = synth.Workload("b", 64, 128e-6, 1400.0, -4.0, n, 1, 0.0, 20.0, boxcar_max, False, "")
    _compare(b.data, 1, w, False, detect_thresh=3.0)


def test_constant_input(hdb, oracle_lib):
    """An RMS of zero: every normalised sample is not a number."""
    n = 16000
    w = synth.Workload("b", 64, 128e-6, 1400.0, -4.0, n, 1, 0.0, 20.0, 64, False, "")
    _compare(np.full((n, 64), 50, np.uint8), 1, w, False)
