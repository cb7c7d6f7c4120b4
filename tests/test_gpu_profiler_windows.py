"""The candidate profiler's windows and stages at their edges, against the
oracle: windows that end inside or start past the last sample, channel counts
around the 256-channel tables and the 32-channel copy tiles, scrunch groups of
one and of many channels (more than a warp's stage holds), odd window sizes,
and a window per candidate of very different widths in one call."""
import numpy as np
import pytest

import heimdall_multibeam_b200 as H
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nchans,fscrunch,out_n,out_d,do_filter", [
    (16, 1, 7, 5, False), (36, 4, 33, 3, True), (260, 260, 64, 9, False), (264, 33, 16, 8, True),
    (512, 1, 9, 4, False), (8192, 8192, 10, 2, False),
])
def test_profiler_edges(hdb, oracle_lib, nchans, fscrunch, out_n, out_d, do_filter):
    rng = np.random.default_rng(nchans + out_n)
    nsamps, dt, f0, bw = 4001 if nchans < 8000 else 601, 128e-6, 1500.0, 300.0
    df = -bw / nchans
    fb = rng.integers(0, 256, size=(nsamps, nchans), dtype=np.uint8)
    dms = oracle.dm_list(0.0, 60.0, dt, 40.0, f0, df, nchans, 1.25)
    last = len(dms) - 1
    reqs = [(0, 0, 0), (nsamps // 2, 5, last // 2), (nsamps - 1, 2, last), (nsamps + 500, 0, 1),
            (nsamps // 3, 9, last)]
    if nchans > 4000:
        reqs = reqs[:3]
    got = H.profile_candidates(fb, dt, f0, df, dms, reqs, out_n, out_d, fscrunch, do_filter)
    for (samp, filt, dm_idx), g in zip(reqs, got):
        r = oracle.profile(fb, dt, f0, df, dms, samp, filt, dm_idx, out_n, out_d, fscrunch,
                           do_filter)
        for k in ("dm_time", "dm0_time", "freq_time"):
            a, b = np.asarray(g[k], np.float32), np.asarray(r[k], np.float32).reshape(g[k].shape)
            np.testing.assert_array_equal(np.isnan(a), np.isnan(b), err_msg=k)
            m = ~np.isnan(a)
            np.testing.assert_array_equal(a[m].view(np.uint32), b[m].view(np.uint32),
                                          err_msg=f"{k} samp {samp} filter {filt}")


@pytest.mark.parametrize("filt,out_n", [(12, 4), (15, 4), (16, 3)])
def test_freq_time_sums_past_exact_integers(hdb, oracle_lib, filt, out_n):
    """Bins of 2^(filt - 2) samples x 16 channels of bytes near 255: sums below
    2^24 (integer adds) and above (the float adds in the reference's order)."""
    rng = np.random.default_rng(filt)
    nchans, nsamps = 32, out_n << filt
    fb = rng.integers(200, 256, size=(nsamps, nchans), dtype=np.uint8)
    dms = np.array([0.0, 1.0], np.float32)
    g = H.profile_candidates(fb, 64e-6, 1500.0, -1.0, dms, [(nsamps // 2, filt, 0)], out_n, 1, 16)[0]
    r = oracle.profile(fb, 64e-6, 1500.0, -1.0, dms, nsamps // 2, filt, 0, out_n, 1, 16, False)
    a, b = g["freq_time"], np.asarray(r["freq_time"], np.float32).reshape(g["freq_time"].shape)
    np.testing.assert_array_equal(np.isnan(a), np.isnan(b))
    m = ~np.isnan(a)
    np.testing.assert_array_equal(a[m].view(np.uint32), b[m].view(np.uint32))


def test_profiler_calls_from_threads_at_once(hdb):
    """Calls of different sizes from several threads, each with its own
    workspace: every answer equals the one a lone call gives."""
    from concurrent.futures import ThreadPoolExecutor
    rng = np.random.default_rng(1)
    dms = np.linspace(0.0, 50.0, 20).astype(np.float32)
    work = []
    for k in range(6):
        fb = rng.integers(0, 256, size=(3000 + 1000 * k, 64), dtype=np.uint8)
        work.append((fb, [(500 + 100 * k, k, 5 + k), (1500, 2, 3)]))

    def one(w):
        return H.profile_candidates(w[0], 128e-6, 1400.0, -4.0, dms, w[1], 32, 8, 16)

    want = [one(w) for w in work]
    with ThreadPoolExecutor(4) as ex:
        for got in (list(ex.map(one, work)) for _ in range(5)):
            for a, b in zip(got, want):
                for p, q in zip(a, b):
                    for k in ("dm_time", "dm0_time", "freq_time", "snr_dm"):
                        np.testing.assert_array_equal(p[k].view(np.uint32), q[k].view(np.uint32))
