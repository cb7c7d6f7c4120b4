"""Several time-scrunched widths in searches large enough for the tiles to be
selected by the boxcars' maxima (test_gpu_hit_tiles has at most two): more of
them than keep maxima, so that the selection skips some widths' tiles and counts
others' in full; and series whose RMS is zero, whose bound no maximum can be
held against.  Candidates and giants equal the oracle's bit for bit."""
import os
import sys

import numpy as np
import pytest

import heimdall_multibeam_b200 as H
from heimdall_multibeam_b200 import synth

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from test_gpu_parity import _compare  # noqa: E402

pytestmark = pytest.mark.gpu

TS_GMAX = 4  # time-scrunched widths that keep maxima
NCH, DT, F0, DF, DM = 64, 128e-6, 1400.0, -4.0, 40.0


def _workload(nsamps, boxcar_max):
    tiles = (nsamps - int(synth.max_delay_samples(DM, NCH, DT, F0, DF)) - boxcar_max) // 2048
    assert len(H.dm_list_guru(0.0, DM, DT, 40.0, F0, DF, NCH, 1.25)) * tiles > 148 * 8
    return synth.Workload("s", NCH, DT, F0, DF, nsamps, 1, 0.0, DM, boxcar_max, False, "")


@pytest.mark.parametrize("boxcar_max,min_ts", [(512, 64), (1024, 8), (2048, 64), (4096, 4096)])
def test_scrunched_widths_selected(hdb, oracle_lib, boxcar_max, min_ts):
    w = _workload(56011, boxcar_max)
    scrunched = [b for b in (1 << k for k in range(13)) if min_ts <= b <= boxcar_max]
    assert len(scrunched) > TS_GMAX or (boxcar_max, min_ts) in ((512, 64), (4096, 4096))
    pulses = [synth.Pulse(7000.0, 20.0, 1e-3, 30.0), synth.Pulse(23456.0, 35.0, 6e-3, 25.0),
              synth.Pulse(41000.0, 30.0, boxcar_max * DT / 2, 40.0)]
    b = synth.make_beam(w.nsamps, NCH, DT, F0, DF, pulses, seed=boxcar_max + min_ts)
    assert len(_compare(b.data, 1, w, False, min_tscrunch_width=min_ts)) >= 2


@pytest.mark.parametrize("min_ts", [4096, 8])
@pytest.mark.parametrize("what", ["constant", "spikes"])
def test_zero_rms_selected(hdb, oracle_lib, what, min_ts):
    w = _workload(56011, 256)
    fb = np.full((w.nsamps, NCH), 50, np.uint8)
    if what == "spikes":  # the median of magnitudes stays zero
        fb[5000::9000] = 90
    _compare(fb, 1, w, False, min_tscrunch_width=min_ts)
