"""Thresholding by the tiles that the boxcars' maxima leave: enough tiles for the
selection to be made, pulses at tile ends, at the ends of the 800-sample
stretches and of the 3125-sample groups, in the incomplete last group and none
at all, with and without time-scrunched widths: candidates and giants equal the
oracle's bit for bit."""
import os
import sys

import pytest

import heimdall_multibeam_b200 as H
from heimdall_multibeam_b200 import synth

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from test_gpu_parity import _compare  # noqa: E402

pytestmark = pytest.mark.gpu

EDGES = {"tiles": (2047, 2048, 4095, 40960), "stretches": (799, 800, 3125 * 7 + 2400, 3125 * 9 + 799),
         "groups": (3124, 3125, 3125 * 19, 3125 * 20 - 1), "rest": (22 * 3125 + 5, 22 * 3125 + 900),
         "none": ()}


@pytest.mark.parametrize("min_ts", [4096, 256])
@pytest.mark.parametrize("where", sorted(EDGES))
def test_selected_tiles(hdb, oracle_lib, where, min_ts):
    dt, f0, df, nch, dm_max, bmax = 128e-6, 1400.0, -4.0, 64, 300.0, 512
    n = 22 * 3125 + 1100 + bmax + int(synth.max_delay_samples(dm_max, nch, dt, f0, df))
    pulses = [synth.Pulse(float(t + bmax // 2), 40.0 * k, (2e-4, 3e-2)[k % 2], 30.0)
              for k, t in enumerate(EDGES[where])]
    b = synth.make_beam(n, nch, dt, f0, df, pulses, seed=5)
    assert len(H.dm_list_guru(0.0, dm_max, dt, 40.0, f0, df, nch, 1.25)) * 34 > 148 * 8
    w = synth.Workload("t", nch, dt, f0, df, n, 1, 0.0, dm_max, bmax, False, "")
    cands = _compare(b.data, 1, w, False, min_tscrunch_width=min_ts)
    assert where == "none" or len(cands) >= 1
