"""Normalise + prefix sum with more time-concatenated beams than a block's RMS
table in shared memory holds for 8 series, and a last block of fewer series,
whose own values would fit: every block of the launch divides by the values in
global memory.  The last filterbanks, whose trials that block holds, give the
oracle's candidates and giants."""
import numpy as np
import pytest

import heimdall_multibeam_b200 as H
import oracle
from heimdall_multibeam_b200 import synth

pytestmark = pytest.mark.gpu


def test_many_beams_and_a_short_last_block(hdb, oracle_lib):
    nchans, dt, f0, df, nbeams, stride, units = 32, 256e-6, 1400.0, -2.0, 260, 120, 113
    kw = dict(dt=dt, f0=f0, df=df, dm_min=0.0, dm_max=100.0, boxcar_max=16, baseline_length=0.01)
    trials = len(H.dm_list_guru(0.0, 100.0, dt, 40.0, f0, df, nchans, 1.25))
    nser = units * trials
    # 8 series a block; the table of 8 does not fit, that of the last block would
    assert nser >= 8 * 295 + 1 and nser % 8
    assert 8 * nbeams > 2048 >= (nser % 8) * nbeams
    nsamps = nbeams * stride
    quiet = synth.make_beam(nsamps, nchans, dt, f0, df, [], seed=40).data
    loud = [synth.make_beam(nsamps, nchans, dt, f0, df,
                            [synth.Pulse(float(k * stride + 4), 60.0 + 10.0 * (k % 5), 5e-4, 40.0)
                             for k in range(u, nbeams - 1, 13)], seed=41 + u, beam=u).data
            for u in range(2)]
    fbs = [quiet] * (units - 2) + loud
    with H.Pipeline(H.default_params(nchans=nchans, output_dir=None, **kw),
                    cleaning=False) as pl:
        pl.execute_beams(fbs, nbeams=nbeams)
        g = pl.giants()
        got = [H.cand_lines(pl.candidates(u)) for u in (0, units - 2, units - 1)]
    end = len(g["peaks"])
    for k, u in ((2, units - 1), (1, units - 2), (0, 0)):
        r = oracle.execute(fbs[u], nbeams=nbeams, clean=0, **kw)
        want = oracle.cand_lines(r["groups"], nsamps, nbeams, 0, r["nsamps_processed"], 16, dt,
                                 beam=u * nbeams)
        assert got[k] == want, u
        n = len(r["giants"]["peaks"])
        assert n >= 10 or u == 0
        if u:
            np.testing.assert_array_equal(g["peaks"][end - n:end].view(np.uint32),
                                          r["giants"]["peaks"].view(np.uint32))
            np.testing.assert_array_equal(g["inds"][end - n:end], r["giants"]["inds"])
            end -= n
