"""Zapped rows beside kept ones in the cleaning's transpose: channel counts with
and without whole 16-byte rows, below and above one tile of 128 channels, sample
counts that end inside a tile, dense bursts: candidates and giants equal the
oracle's bit for bit."""
import os
import sys

import numpy as np
import pytest

import heimdall_multibeam_b200 as H
from heimdall_multibeam_b200 import synth

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from test_gpu_parity import _compare  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nch", [16, 36, 132, 160])
@pytest.mark.parametrize("n", [16000, 16129])
def test_masked_rows(hdb, oracle_lib, nch, n):
    w = synth.Workload("z", nch, 256e-6, 1400.0, -240.0 / nch, n, 1, 0.0, 40.0, 64, True, "")
    b = synth.make_beam(n, nch, w.dt, w.f0, w.df, [synth.Pulse(9000.0, 30.0, 1e-3, 40.0)],
                        seed=nch + n)
    fb = np.array(b.data)
    rng = np.random.default_rng(n + nch)
    for t in rng.integers(0, n, 40):          # bursts of one to nine spectra
        e = int(t) + int(rng.integers(1, 10))
        fb[t:e] = np.minimum(fb[t:e].astype(int) + 60, 255).astype(np.uint8)
    fb[-3:] = 255                              # the last spectra too
    _compare(fb, 1, w, True, baseline_length=0.5)
