"""Single gulps served by the CUDA graph (hd_execute, hd_execute_device): from new
host and device buffers each time, with packed samples, cleaning and
time-concatenated beams: each gulp gives what the host-sized path gives."""
import numpy as np
import pytest

import heimdall_multibeam_b200 as H
from heimdall_multibeam_b200 import synth

pytestmark = pytest.mark.gpu


def _gulps(nbits, nbeams, n=3):
    out = []
    for k in range(n):
        beams = [synth.make_beam(12001, 64, 256e-6, 1400.0, -4.0,
                                 [synth.Pulse(3000.0 + 500 * k, 20.0, 1e-3, 40.0),
                                  synth.Pulse(8000.0, 35.0, 4e-3, 40.0)], seed=10 * k + b, beam=b)
                 for b in range(nbeams)]
        fb = np.asarray(synth.stf(beams)) if nbeams > 1 else np.array(beams[0].data)
        if nbits < 8:
            fb = np.clip((fb.astype(int) - 60) >> (8 - nbits - 1), 0, (1 << nbits) - 1)
            fb = synth.pack_filterbank(fb.astype(np.uint16), nbits)
        out.append(np.ascontiguousarray(fb))
    return out


@pytest.mark.parametrize("nbits,clean,nbeams", [(8, False, 1), (8, True, 1), (8, True, 2),
                                                (4, False, 1), (2, True, 1), (1, False, 1)])
@pytest.mark.parametrize("device", [False, True])
def test_single_gulps_replay(hdb, device, nbits, clean, nbeams):
    torch = pytest.importorskip("torch")
    p = H.default_params(nchans=64, dt=256e-6, f0=1400.0, df=-4.0, dm_max=40.0, boxcar_max=64,
                         output_dir=None)

    def run(graphs):
        res = []
        with H.Pipeline(p, cleaning=clean) as pl:
            pl.set_graphs(graphs)
            for fb in _gulps(nbits, nbeams):
                if device:
                    d = torch.from_numpy(fb.view(np.uint8)).cuda()
                    err, proc = pl.execute_device(d.data_ptr(), fb.shape[0], nbeams=nbeams,
                                                  nbits=nbits)
                else:
                    err, proc = pl.execute(fb, nbeams=nbeams, nbits=nbits, raise_on_error=False)
                g = pl.giants()
                res.append((err, proc, H.cand_lines(pl.candidates()),
                            {k: np.asarray(v).copy() for k, v in g.items()}))
            return res, pl.graph_replays()

    (got, replays), (want, none) = run(True), run(False)
    # (packed samples with cleaning are refused, by both)
    refused = clean and nbits < 8
    assert none == 0 and (replays == 0 if refused else replays >= 1)
    assert all((r[0] == H.HD_INVALID_NBITS) == refused for r in want)
    for a, b in zip(got, want):
        assert a[:3] == b[:3]
        for k in b[3]:
            np.testing.assert_array_equal(a[3][k].view(np.uint8), b[3][k].view(np.uint8), err_msg=k)
    # (the cleaning takes pulses of this low a DM for interference)
    assert any(len(r[2]) for r in want) or nbits < 8 or clean
