"""Several time-scrunched widths in one search (min_tscrunch_width below the
widest boxcar): their block-RMS windows end in stale values of earlier widths,
their tiles are skipped where the group maxima stay below the threshold, and
more of them than keep maxima (TS_GMAX) are counted in full.  Giants (peak
bits, indices), labels and .cand lines equal the oracle's, for one beam (with
the maxima) and for a beam pair (without)."""
import os
import sys

import numpy as np
import pytest

import heimdall_multibeam_b200 as H
import oracle
from heimdall_multibeam_b200 import synth

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from test_gpu_parity import _compare  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbeams", [1, 2])
@pytest.mark.parametrize("boxcar_max,min_ts", [(64, 64), (512, 64), (1024, 8), (2048, 1024)])
def test_scrunched_widths(hdb, oracle_lib, nbeams, boxcar_max, min_ts):
    w = synth.Workload("ts", 64, 128e-6, 1400.0, -4.0, 20011, nbeams, 0.0, 40.0, boxcar_max, False,
                       "")
    beams = [synth.make_beam(w.nsamps, w.nchans, w.dt, w.f0, w.df,
                             [synth.Pulse(4000.0, 20.0, 1e-3, 30.0),
                              synth.Pulse(9000.0 + 700 * b, 30.0, boxcar_max * w.dt / 2, 40.0)],
                             seed=17 + b, beam=b) for b in range(nbeams)]
    cands = _compare(synth.stf(beams), nbeams, w, False, min_tscrunch_width=min_ts)
    assert len(cands) >= 2
