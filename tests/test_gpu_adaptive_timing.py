"""Stage times of a gulp at adaptive time resolution (hd_get_timing): the
stages of all scrunch groups add up to the whole gulp, and the time of the
series does not hold the groups' searches, which a low threshold makes long."""
import numpy as np
import pytest

import heimdall_multibeam_b200 as H
from heimdall_multibeam_b200 import synth

pytestmark = pytest.mark.gpu


def test_stages_of_all_groups(hdb):
    w = synth.SEARCH_C0
    p = H.default_params(nchans=w.nchans, dt=w.dt, f0=w.f0, df=w.df, dm_min=w.dm_min,
                         dm_max=w.dm_max, boxcar_max=w.boxcar_max, output_dir=None,
                         use_scrunching=True, detect_thresh=2.0, max_giant_rate=1000.0)
    fb = synth.make_c0().data
    ratio = []
    with H.Pipeline(p, cleaning=False) as pl:
        for _ in range(4):
            # (so many events that clustering is left out)
            assert pl.execute(fb, raise_on_error=False)[0] == H.HD_TOO_MANY_EVENTS
            t = pl.timing()
            stages = sum(v for k, v in t.items() if k != "total")
            assert abs(stages - t["total"]) <= 0.02 * t["total"] + 0.05, t
            ratio.append(t["baseline_scan"] / (t["boxcar_threshold"] + t["giants"]))
    assert np.median(ratio[1:]) < 0.5, ratio
