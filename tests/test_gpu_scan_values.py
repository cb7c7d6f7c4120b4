"""Prefix sums over series whose samples are exact zeros for whole stages
(which the divisions' fast path does not take), beside stages of ordinary
values, at lengths around the stages' 512 samples: candidates and giants equal
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


@pytest.mark.parametrize("extra", [0, 1, 2, 3, 511])
def test_zero_stretches(hdb, oracle_lib, extra):
    w = synth.Workload("z", 64, 128e-6, 1400.0, -4.0, 20480, 1, 0.0, 40.0, 256, False, "")
    lost = int(synth.max_delay_samples(w.dm_max, w.nchans, w.dt, w.f0, w.df))
    n = 20480 + lost + extra  # series of about 40 stages and `extra` samples
    b = synth.make_beam(n, w.nchans, w.dt, w.f0, w.df,
                        [synth.Pulse(3000.0, 20.0, 1e-3, 40.0),
                         synth.Pulse(17000.0, 30.0, 4e-3, 40.0)], seed=31)
    fb = np.array(b.data)
    fb[6000:12000] = 96          # a constant input: zeros after the baseline
    fb[14000:14100] = 0
    w = synth.Workload("z", 64, 128e-6, 1400.0, -4.0, n, 1, 0.0, 40.0, 256, False, "")
    cands = _compare(fb, 1, w, False, baseline_length=0.05)
    assert len(cands) >= 2
