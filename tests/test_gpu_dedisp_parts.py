"""Dedispersion whose four-sample words do not all fit the device: a few
filterbanks, or of one filterbank a few channels, at a time, the channels' sums
meeting in the output.  The sums are whole numbers and equal the oracle's; a
gulp that leaves no room for the words gives what it gives with room."""
import os
import sys

import numpy as np
import pytest

import heimdall_multibeam_b200 as H
import oracle
from heimdall_multibeam_b200 import synth

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from device_room import device_room  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chans_at_once", [1, 3, 100, 257, 600])
@pytest.mark.parametrize("nchans", [4, 260, 776])
@pytest.mark.parametrize("tune", ["0", "1"])
def test_channels_in_parts(hdb, oracle_lib, monkeypatch, nchans, chans_at_once, tune):
    dt, f0, df = 256e-6, 1400.0, -200.0 / nchans
    dms = np.linspace(0.0, 60.0, 11).astype(np.float32)
    table = oracle.delay_table(nchans, dt, f0, df)
    md = int(oracle.delays(dms, table).max())
    nsamps = md + 2333
    # a channel's words are between split + md and that and a tile more
    monkeypatch.setenv("HDB_DEDISP_WORDS", str(chans_at_once * (640 + md + 2600)))
    monkeypatch.setenv("HDB_DEDISP_TUNE", tune)
    monkeypatch.setenv("HDB_TUNE_CACHE", "0")
    full = np.full((nsamps, nchans), 255, np.uint8)
    some = np.random.default_rng(nchans).integers(0, 256, size=(nsamps, nchans), dtype=np.uint8)
    gaps = np.ones(nchans, np.int32)
    gaps[:nchans // 3] = 0           # whole parts without a channel
    gaps[nchans // 2::5] = 0
    gaps[-nchans // 4:] = 0
    for fb, km in ((full, None), (some, gaps), (some, None)):
        plan = H.DedispPlan(nchans, dt, f0, df)
        plan.set_dm_list(dms)
        if km is not None:
            plan.set_killmask(km)
        np.testing.assert_array_equal(plan.execute(fb), oracle.dedisperse(fb, dms, table, km))


# filterbanks' worth of words: two and a half of the five, and a third of one
@pytest.mark.parametrize("share", [2.5, 0.33])
@pytest.mark.parametrize("adaptive", [False, True])
def test_filterbanks_in_parts(hdb, monkeypatch, share, adaptive):
    torch = pytest.importorskip("torch")
    w = synth.Workload("p", 64, 256e-6, 1400.0, -4.0, 20011, 5, 0.0, 300.0, 256, False, "")
    p = H.default_params(nchans=w.nchans, dt=w.dt, f0=w.f0, df=w.df, dm_max=w.dm_max,
                         boxcar_max=w.boxcar_max, output_dir=None, use_scrunching=adaptive)
    beams = [torch.from_numpy(b.data).cuda() for b in synth.make_multibeam(w, seed=9, snr_lo=12)]
    md = int(synth.max_delay_samples(w.dm_max, w.nchans, w.dt, w.f0, w.df)) + 1

    def run():
        out = []
        with H.Pipeline(p, cleaning=False) as pl:
            for _ in range(3):  # the third is a graph's replay at native resolution
                err, _, st = pl.execute_beams([b.data_ptr() for b in beams], nsamps=w.nsamps,
                                              on_device=True)
                g = pl.giants()
                out.append((err, st, [H.cand_lines(pl.candidates(u)) for u in range(5)],
                            {k: np.asarray(v).tolist() for k, v in g.items()}))
            return out, pl.graph_replays()

    want, replays = run()
    words = w.nchans * ((w.nsamps - md) // 4 + md + 400)
    monkeypatch.setenv("HDB_DEDISP_WORDS", str(int(share * words)))
    got, again = run()
    assert got == want and again == replays == (0 if adaptive else 2)
    assert sum(len(c) for c in want[0][2]) >= 5


@pytest.mark.parametrize("units,nchans,nsamps", [(1, 1024, 1 << 16), (6, 256, 1 << 16)])
def test_gulp_without_room_for_its_words(hdb, units, nchans, nsamps):
    """The words of these gulps are the largest part of what they need (few
    trials, long delays)."""
    torch = pytest.importorskip("torch")
    dt, f0, df = 64e-6, 1400.0, -400.0 / nchans
    w = synth.Workload("m", nchans, dt, f0, df, nsamps, units, 980.0, 1000.0, 64, False, "")
    md = int(synth.max_delay_samples(w.dm_max, nchans, dt, f0, df)) + 1
    assert md < nsamps // 2
    p = H.default_params(nchans=nchans, dt=dt, f0=f0, df=df, dm_min=w.dm_min, dm_max=w.dm_max,
                         boxcar_max=64, output_dir=None)
    beams = [torch.from_numpy(
        synth.make_beam(nsamps, nchans, dt, f0, df, [synth.Pulse(9000.0, 990.0, 1e-3, 40.0)],
                        seed=77 + u, beam=u).data).cuda() for u in range(units)]
    words = 4 * units * nchans * ((nsamps - md) // 4 + md)

    def run():
        with H.Pipeline(p, cleaning=False) as pl:
            before = torch.cuda.mem_get_info()[0]
            out = []
            for _ in range(3):
                err, _, st = pl.execute_beams([b.data_ptr() for b in beams], nsamps=nsamps,
                                              on_device=True, raise_on_error=False)
                out.append((err, st, [H.cand_lines(pl.candidates(u)) for u in range(units)]))
            return out, before - torch.cuda.mem_get_info()[0]

    want, used = run()
    want, used = run()  # (what the first call loads and tunes stays)
    assert want[0][0] == H.HD_NO_ERROR and all(len(c) for c in want[0][2])
    assert words > (64 << 20) and used > words
    with device_room(torch, used - words // 2):
        got, less = run()
    assert got == want
    assert less < used - words // 3
