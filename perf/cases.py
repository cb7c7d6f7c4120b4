"""The calls whose speed matters, as a user's program makes them.

Each case is one call (or one short run of calls) through the package's public
entry points: whole gulps searched in the forms an observatory runs them
(plain, survey size with cleaning, batched multibeam from device and from host
memory, time-concatenated beams at adaptive time resolution, packed samples,
beams of uneven shapes), the dedispersion plan on its own, and what follows a
search (scoring candidates, one training step, profiling candidates).
`listed()` holds the named shapes, `draw()` others of the same ranges."""
import math
import os
import random

import numpy as np
import torch

import heimdall_multibeam_b200 as H
from heimdall_multibeam_b200 import synth

DEV = "cuda"
REALS = ("snr", "time", "dm")
WHOLE = ("samp_idx", "filter", "dm_trial", "members", "begin", "end", "beam")


# --------------------------------------------------------------------------
# The cases
# --------------------------------------------------------------------------
def gulp(name, nchans, nsamps, dt_us, f0, bw, dm_max, boxcar_max, beams=1, units=1,
         cleaning=False, adaptive=False, nbits=8, source="host", pulses=3):
    c = dict(kind="gulp", nchans=nchans, nsamps=nsamps, dt_us=dt_us, f0=f0, bw=bw, dm_max=dm_max,
             boxcar_max=boxcar_max, beams=beams, units=units, cleaning=cleaning,
             adaptive=adaptive, nbits=nbits, source=source, pulses=pulses)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a quick-look search of a short narrow-band gulp: launches and host round trips count
        gulp("small_gulp", 64, 8192, 655.36, 851.0, 25.0, 600.0, 256),
        # the plain single-beam search, filterbank in ordinary host memory (hd_execute)
        gulp("plain_host", 256, 1 << 16, 64.0, 1500.0, 400.0, 1000.0, 1024),
        # one beam of a survey receiver with RFI cleaning, filterbank already on the GPU
        gulp("survey_device", 1024, 1 << 18, 64.0, 1520.0, 400.0, 2000.0, 4096, cleaning=True,
             source="device", pulses=20),
        # a multibeam receiver's gulp, all beams in one call, filterbanks on the GPU
        gulp("multibeam_device", 320, 1 << 15, 655.36, 851.0, 31.25, 2000.0, 512, units=36,
             source="device", pulses=2),
        # the same gulp handed over in page-locked host memory
        gulp("multibeam_host", 320, 1 << 15, 655.36, 851.0, 31.25, 2000.0, 512, units=36,
             source="pinned", pulses=2),
        # four beams concatenated in time, cleaned, at adaptive time resolution (the defaults)
        gulp("stf_adaptive", 256, 1 << 16, 64.0, 1500.0, 400.0, 1000.0, 1024, beams=4,
             cleaning=True, adaptive=True, source="device"),
        # 2-bit digitised data, as archives hold it, with a length that is no round number
        gulp("packed_2bit", 512, 100003, 128.0, 1520.0, 300.0, 800.0, 2048, nbits=2),
        # beams of different channel counts, lengths and DM ranges in one call
        dict(name="uneven_set", kind="set", nbeams=12, shapes_seed=2027, log2_max=17),
        # the dedispersion plan alone, device pointers (dedisp_execute_adv)
        dict(name="dedisp_device", kind="dedisp", nchans=256, nsamps=1 << 16, dt_us=64.0,
             f0=1500.0, bw=400.0, dm_max=1000.0, nbits=8),
        # scoring a long candidate list whose patches are on the GPU
        dict(name="classify", kind="classify", n=4096),
        # one training step of the classifier: loss and gradients of a batch
        dict(name="gradients", kind="gradients", n=128),
        # plots of a gulp's candidates: the profiler on a filterbank on the GPU
        dict(name="profile", kind="profile", nchans=256, nsamps=1 << 16, n=12, out_nsamps=64,
             out_dms=32, fscrunch=16, do_filter=False),
    ]


# candidates of one beam that a pass has room for
ROOM = 1024
# multiply-adds of the largest search drawn: that of the survey gulp
MOST_ADDS = 3.0e11


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def dm_trials(nchans, dt, f0, df, dm_max):
    """DM list of the library's spacing rule (smearing tolerance 1.25, pulse width 40 us; times in
    microseconds, frequencies in GHz, every trial stored in 32 bits)."""
    f = (f0 + ((nchans // 2) - 0.5) * df) * 1e-3
    a2 = (8.3 * df / f ** 3) ** 2
    b2 = a2 * nchans * nchans / 16.0
    c = ((dt * 1e6) ** 2 + 1600.0) * (1.25 ** 2 - 1.0)
    out = [np.float32(0.0)]
    while out[-1] < dm_max:
        p = float(out[-1])
        k = c + 1.25 ** 2 * a2 * p * p
        out.append(np.float32((b2 * p + math.sqrt(-a2 * b2 * p * p + (a2 + b2) * k)) / (a2 + b2)))
    return np.array(out, np.float32)


def fit_dm(c, nsamps, boxcar_max, copies, most_adds=MOST_ADDS):
    """Halves the DM range until the delays leave room in the gulp and the work is bounded."""
    dt, df = c["dt_us"] * 1e-6, -c["bw"] / c["nchans"]
    while c["dm_max"] > 2.0:
        md = synth.max_delay_samples(c["dm_max"], c["nchans"], dt, c["f0"], df)
        if md + boxcar_max < 0.6 * nsamps:
            trials = len(dm_trials(c["nchans"], dt, c["f0"], df, c["dm_max"]))
            if trials * copies < 60000 and trials * c["nchans"] * (nsamps - md) * copies < most_adds:
                break
        c["dm_max"] = round(c["dm_max"] / 2, 3)
    return c


def band(rng):
    f0 = round(rng.uniform(700.0, 1600.0), 3)
    return f0, round(f0 * rng.uniform(0.05, 0.28), 3)


def draw(rng):
    kind = rng.choice(("one", "one", "one", "beams", "beams", "stf", "packed", "set", "dedisp",
                       "dedisp", "classify", "gradients", "profile"))
    if kind == "set":
        return dict(kind="set", nbeams=rng.randint(3, 10), shapes_seed=rng.randint(1, 10 ** 6),
                    log2_max=rng.choice((15, 16)))
    if kind == "classify":
        return dict(kind="classify", n=log_int(rng, 1, 4096))
    if kind == "gradients":
        return dict(kind="gradients", n=log_int(rng, 8, 128))
    f0, bw = band(rng)
    dt_us = rng.choice((64.0, 128.0, 327.68, 655.36))
    dm_max = rng.choice((100.0, 300.0, 500.0, 1000.0, 2000.0))
    if kind == "profile":
        fs = rng.choice((4, 8, 16))
        return dict(kind="profile", nchans=fs * rng.randint(8, 16), nsamps=log_int(rng, 20000, 60000),
                    n=rng.randint(1, 12), out_nsamps=rng.choice((32, 64)),
                    out_dms=rng.choice((16, 24, 32)), fscrunch=fs, do_filter=rng.random() < 0.5)
    if kind == "dedisp":
        c = dict(kind="dedisp", nchans=4 * log_int(rng, 8, 256), nsamps=log_int(rng, 6000, 120000),
                 dt_us=dt_us, f0=f0, bw=bw, dm_max=dm_max, nbits=rng.choice((8, 8, 8, 16)))
        return fit_dm(c, c["nsamps"], 0, 1, 3.0e10)
    boxcar_max = 2 ** rng.randint(5, 12)
    nchans, nsamps, beams, units, cleaning, adaptive, nbits = 4 * log_int(rng, 8, 256), 0, 1, 1, rng.random() < 0.5, False, 8
    source = rng.choice(("host", "device", "device"))
    if kind == "one":
        nsamps = log_int(rng, 8000, 250000)
        adaptive = rng.random() < 0.2
    elif kind == "beams":
        units = log_int(rng, 3, 36)
        nchans = 4 * log_int(rng, 16, 100)
        nsamps = log_int(rng, 8000, 32768)
        source = rng.choice(("pinned", "device", "device"))
        boxcar_max = min(boxcar_max, 1024)
    elif kind == "stf":
        beams = rng.randint(2, 5)
        nchans = 4 * log_int(rng, 16, 80)
        nsamps = log_int(rng, 8000, 50000)
        adaptive = rng.random() < 0.5
    else:
        nbits = rng.choice((2, 4, 16))
        nchans = 32 * log_int(rng, 2, 24)
        nsamps = log_int(rng, 10000, 100000)
        cleaning = False
    boxcar_max = min(boxcar_max, 2 ** int(math.log2(nsamps / 4)))
    c = gulp(None, nchans, nsamps, dt_us, f0, bw, dm_max, boxcar_max, beams, units, cleaning,
             adaptive, nbits, source, rng.randint(1, 4))
    return fit_dm(c, nsamps, boxcar_max, beams * units, MOST_ADDS if kind == "one" else 8e10)


# --------------------------------------------------------------------------
# Inputs: noise (mean 128, sd 16), dispersed pulses, RFI where it is cleaned
# --------------------------------------------------------------------------
def filterbank(rnd, gen, nsamps, nchans, dt, f0, df, dm_max, boxcar_max, pulses, rfi):
    """One beam's (nsamps, nchans) uint8 filterbank on the GPU."""
    x = torch.randn((nsamps, nchans), generator=gen, device=DEV)
    x.mul_(16.0).add_(128.0)
    md = synth.max_delay_samples(dm_max, nchans, dt, f0, df)
    hi = max(nsamps - md - 2 * boxcar_max, boxcar_max + 1)
    for _ in range(pulses):
        p = synth.Pulse(rnd.uniform(boxcar_max, hi), rnd.uniform(min(50.0, dm_max / 2), dm_max),
                        math.exp(rnd.uniform(math.log(max(1e-4, dt)), math.log(max(3e-2, 4 * dt)))),
                        rnd.uniform(8.0, 40.0))
        synth.inject_pulse_device(torch, x, p, dt, f0, df)
    if rfi:  # 5 % of the channels saturated, a few zero-DM bursts
        x[:, rnd.sample(range(nchans), max(1, nchans // 20))] += 640.0
        for _ in range(max(1, nsamps * 10 >> 18)):
            at = rnd.randrange(nsamps - 60)
            x[at:at + rnd.randint(1, 50)] += 128.0
    return x.round_().clamp_(0, 255).to(torch.uint8)


def pack(x, nbits):
    """uint8 samples to packed rows of nbits-bit ones (the top bits), or to 16-bit ones."""
    if nbits == 16:
        return (x.to(torch.int32) * 97 + 11).to(torch.int16).view(torch.uint8)
    v = (x >> (8 - nbits)).view(x.shape[0], -1, 8 // nbits)
    return sum(v[:, :, k] << (k * nbits) for k in range(8 // nbits)).to(torch.uint8).contiguous()


def params(nchans, dt, f0, df, dm_max, boxcar_max, adaptive=False):
    return H.default_params(nchans=nchans, dt=dt, f0=f0, df=df, dm_min=0.0, dm_max=dm_max,
                            boxcar_max=boxcar_max, use_scrunching=adaptive, output_dir=None)


def patches(c, gen):
    """Candidates' normalised DM-time and frequency-time patches: noise rows, every other one with
    a pulse."""
    n = c["n"]
    dm = torch.randn((n, 64, 64), generator=gen, device=DEV)
    ft = torch.randn((n, 64, 256), generator=gen, device=DEV)
    t = torch.arange(64, device=DEV) - 32.0
    amp = torch.rand((n, 1, 1), generator=gen, device=DEV) * 12.0
    amp[::2] = 0.0
    width = 1.0 + 6.0 * torch.rand((n, 1, 1), generator=gen, device=DEV)
    dm += amp * torch.exp(-0.5 * ((t[None, None, :] - 0.3 * t[None, :, None]) / width) ** 2) \
        * torch.exp(-0.5 * (t[None, :, None] / 10.0) ** 2)
    u = torch.arange(256, device=DEV) - 128.0
    ft += 0.2 * amp * torch.exp(-0.5 * ((u[None, None, :] - t[None, :, None]) / (2 * width)) ** 2)
    return dm, ft, (amp.view(-1) > 0).to(torch.int32)


def weights():
    return np.load(os.path.join(H.HERE, "classifier_survey.npy"))


def dedisp_input(c, seed):
    rnd, gen = random.Random(seed), torch.Generator(DEV).manual_seed(seed)
    dt, df = c["dt_us"] * 1e-6, -c["bw"] / c["nchans"]
    x = filterbank(rnd, gen, c["nsamps"], c["nchans"], dt, c["f0"], df, c["dm_max"], 64, 3, False)
    return x if c["nbits"] == 8 else pack(x, c["nbits"])


# --------------------------------------------------------------------------
# What a program has in hand before the call
# --------------------------------------------------------------------------
def prepare(case, seed):
    c, kind = case, case["kind"]
    rnd, gen = random.Random(seed), torch.Generator(DEV).manual_seed(seed)
    if kind == "gulp":
        dt, df = c["dt_us"] * 1e-6, -c["bw"] / c["nchans"]
        fbs = []
        for _ in range(c["units"]):
            one = [filterbank(rnd, gen, c["nsamps"], c["nchans"], dt, c["f0"], df, c["dm_max"],
                              c["boxcar_max"], c["pulses"], c["cleaning"])
                   for _ in range(c["beams"])]
            x = one[0] if len(one) == 1 else torch.cat(one)
            fbs.append(x if c["nbits"] == 8 else pack(x, c["nbits"]))
        x = torch.stack(fbs)
        del fbs
        if c["source"] == "pinned":
            x = torch.empty(x.shape, dtype=x.dtype, pin_memory=True).copy_(x)
        elif c["source"] == "host":
            x = x.cpu().numpy()
        pl = H.Pipeline(params(c["nchans"], dt, c["f0"], df, c["dm_max"], c["boxcar_max"],
                               c["adaptive"]), cleaning=c["cleaning"])
        return dict(case=c, x=x, pl=pl)
    if kind == "set":
        ws = synth.uneven_shapes(c["nbeams"], seed=c["shapes_seed"],
                                 nsamps_range=(1 << 14, 1 << c["log2_max"]))
        fbs = [filterbank(rnd, gen, w.nsamps, w.nchans, w.dt, w.f0, w.df, w.dm_max, w.boxcar_max,
                          2, True) for w in ws]
        ps = [params(w.nchans, w.dt, w.f0, w.df, w.dm_max, w.boxcar_max) for w in ws]
        for b, p in enumerate(ps):
            p.beam = b
        return dict(case=c, fbs=fbs, bs=H.BeamSet(ps, workers=4, cleaning=True),
                    nsamps=[w.nsamps for w in ws])
    if kind == "dedisp":
        x = dedisp_input(c, seed)
        dt, df = c["dt_us"] * 1e-6, -c["bw"] / c["nchans"]
        plan = H.DedispPlan(c["nchans"], dt, c["f0"], df)
        dms = dm_trials(c["nchans"], dt, c["f0"], df, c["dm_max"])
        plan.set_dm_list(dms)
        nout = c["nsamps"] - plan.max_delay
        out = torch.zeros((len(dms), (nout + 3) // 4 * 4), device=DEV)
        return dict(case=c, x=x, plan=plan, out=out, nout=nout)
    if kind in ("classify", "gradients"):
        dm, ft, lab = patches(c, gen)
        clf = H.Classifier()
        clf.set_params(weights())
        if kind == "gradients":
            dm, ft, lab = dm.cpu().numpy(), ft.cpu().numpy(), lab.cpu().numpy()
        return dict(case=c, dm=dm, ft=ft, lab=lab, clf=clf)
    dt, f0, df = 64e-6, 1500.0, -400.0 / c["nchans"]
    x = filterbank(rnd, gen, c["nsamps"], c["nchans"], dt, f0, df, 400.0, 256, 3, False)
    dms = dm_trials(c["nchans"], dt, f0, df, 400.0)
    reqs = [(rnd.randrange(c["nsamps"] // 2), 5 * k % 8, rnd.randrange(len(dms)))
            for k in range(c["n"])]
    return dict(case=c, x=x, dms=dms, reqs=reqs, band=(dt, f0, df))


# --------------------------------------------------------------------------
# One pass
# --------------------------------------------------------------------------
def rows(cands, room):
    """The candidate list, in arrays whose size does not depend on how many were found."""
    n = len(cands)
    if n > room:
        raise RuntimeError(f"{n} candidates, and room for {room}")
    reals, whole = np.zeros((room, len(REALS)), np.float32), np.zeros((room, len(WHOLE)), np.int64)
    for k, f in enumerate(REALS):
        reals[:n, k] = cands[f]
    for k, f in enumerate(WHOLE):
        whole[:n, k] = cands[f]
    return dict(found=n, reals=reals, whole=whole)


def run(state):
    s, c = state, state["case"]
    kind = c["kind"]
    if kind == "gulp":
        pl, x = s["pl"], s["x"]
        if c["units"] > 1:
            step = x.stride(0)
            err, done, _ = pl.execute_beams([x.data_ptr() + u * step for u in range(c["units"])],
                                            nsamps=x.shape[1], nbeams=c["beams"],
                                            on_device=c["source"] == "device")
        elif c["source"] == "host":
            err, done = pl.execute(x[0], nbeams=c["beams"], nbits=c["nbits"])
        else:
            err, done = pl.execute_device(x.data_ptr(), x.shape[1], nbeams=c["beams"],
                                          nbits=c["nbits"])
        return dict(rows(pl.candidates(), c["units"] * c["beams"] * ROOM), status=err,
                    processed=done)
    if kind == "set":
        err, st, done = s["bs"].execute([f.data_ptr() for f in s["fbs"]], s["nsamps"],
                                        on_device=True)
        cands = np.concatenate([s["bs"].candidates(b) for b in range(c["nbeams"])])
        return dict(rows(cands, c["nbeams"] * ROOM), status=np.array([err] + st), processed=np.array(done))
    if kind == "dedisp":
        out = s["out"]
        err = H.lib().dedisp_execute_adv(s["plan"]._p, c["nsamps"], s["x"].data_ptr(), c["nbits"],
                                         c["nchans"] * c["nbits"] // 8, out.data_ptr(), 32,
                                         out.shape[1] * 4, H.DEDISP_DEVICE_POINTERS)
        return dict(status=err, series=out[:, :s["nout"]])
    if kind == "classify":
        return s["clf"].score_device(s["dm"].data_ptr(), s["ft"].data_ptr(), c["n"])
    if kind == "gradients":
        return s["clf"].gradients(s["dm"], s["ft"], s["lab"])
    dt, f0, df = s["band"]
    got = H.profile_candidates(s["x"].data_ptr(), dt, f0, df, s["dms"], s["reqs"],
                               c["out_nsamps"], c["out_dms"], c["fscrunch"], c["do_filter"],
                               nsamps=c["nsamps"], nchans=c["nchans"], on_device=True)
    return {k: np.stack([g[k] for g in got])
            for k in ("dm_time", "dm0_time", "freq_time", "snr_dm", "snr_time", "max_idx")}


# --------------------------------------------------------------------------
# What a pass cannot do without: every input read once, every output written
# once, one add per sample, channel and trial (and the filters' over them)
# --------------------------------------------------------------------------
def search_work(nchans, nsamps, dt, f0, df, dm_max, boxcar_max, nbits=8):
    md = synth.max_delay_samples(dm_max, nchans, dt, f0, df)
    nout = max(0.0, nsamps - md)
    trials = len(dm_trials(nchans, dt, f0, df, dm_max))
    return (nsamps * nchans * nbits / 8.0,
            trials * nout * (nchans + 2.0 * (math.log2(boxcar_max) + 1)), trials * nout)


def work(case):
    c, kind = case, case["kind"]
    if kind in ("gulp", "dedisp"):
        b, f, series = search_work(c["nchans"], c["nsamps"], c["dt_us"] * 1e-6, c["f0"],
                                   -c["bw"] / c["nchans"], c["dm_max"], c.get("boxcar_max", 1),
                                   c["nbits"])
        if kind == "dedisp":
            return {"bytes": b + 4 * series, "flops": series * c["nchans"]}
        n = c["units"] * c["beams"]
        return {"bytes": n * b, "flops": n * f}
    if kind == "set":
        ws = synth.uneven_shapes(c["nbeams"], seed=c["shapes_seed"],
                                 nsamps_range=(1 << 14, 1 << c["log2_max"]))
        each = [search_work(w.nchans, w.nsamps, w.dt, w.f0, w.df, w.dm_max, w.boxcar_max)
                for w in ws]
        return {"bytes": sum(e[0] for e in each), "flops": sum(e[1] for e in each)}
    if kind == "classify":
        return {"bytes": c["n"] * (4.0 * 64 * 320 + 4), "flops": c["n"] * 26.87e6}
    if kind == "gradients":
        return {"bytes": c["n"] * 4.0 * 64 * 320 + 8 * 175666, "flops": 3 * c["n"] * 26.87e6}
    row = c["out_nsamps"] * (c["out_dms"] + 6.0 + c["nchans"] // c["fscrunch"]) + c["out_dms"]
    wide = 2 ** 4 * c["out_nsamps"] * c["nchans"]  # a typical width's window
    return {"bytes": c["n"] * (wide + 4 * row), "flops": c["n"] * wide * c["out_dms"]}


# --------------------------------------------------------------------------
# The same in 64 bits, without the library
# --------------------------------------------------------------------------
def exact_dedisp(c, seed):
    """Channel sums at delays of dm * K (f^-2 - f0^-2) / dt + 1/2 cut to whole samples, the delay
    table in 32 bits as the interface documents it."""
    f4 = np.float32
    dt, df = f4(c["dt_us"] * 1e-6), f4(-c["bw"] / c["nchans"])
    dms = dm_trials(c["nchans"], c["dt_us"] * 1e-6, c["f0"], -c["bw"] / c["nchans"], c["dm_max"])
    b = f4(1) / f4(c["f0"])
    a = f4(1) / (f4(c["f0"]) + np.arange(c["nchans"], dtype=f4) * df)
    table = f4(4148.808) * (a * a - b * b) / dt
    delays = np.floor(np.maximum(dms[:, None] * table[None, :] + f4(0.5), f4(0))).astype(np.int64)
    nout = c["nsamps"] - int(delays.max())
    if len(dms) * nout * c["nchans"] > 2.0e10:
        return None
    x = dedisp_input(c, seed)
    if c["nbits"] == 16:
        x = x.view(torch.int16).to(torch.int32) & 0xFFFF
    out = torch.zeros((len(dms), nout), dtype=torch.float64, device=DEV)
    at = torch.from_numpy(delays).to(DEV)
    for ch in range(c["nchans"]):
        row = x[:, ch].to(torch.float64)
        out += row.unfold(0, nout, 1)[at[:, ch]]
    return out


def exact_network(c, seed, train):
    """The two-branch network (3 x 3 convolutions with ReLU and 2 x 2 maxima, two dense layers)."""
    F = torch.nn.functional
    dm, ft, lab = patches(c, torch.Generator(DEV).manual_seed(seed))
    p = torch.from_numpy(weights()).to(DEV).double().requires_grad_(train)
    at = 0

    def take(*shape):
        nonlocal at
        n = math.prod(shape)
        at += n
        return p[at - n:at].view(*shape)

    feats = []
    for x in (dm, ft):
        x = x.double().clamp(-16.0, 16.0)[:, None]
        for ci, co in ((1, 8), (8, 16), (16, 32)):
            w, b = take(co, ci, 3, 3), take(co)
            x = F.max_pool2d(F.relu(F.conv2d(x, w, b, padding=1)), 2)
        feats.append(x.flatten(1))
    x = torch.cat(feats, 1)
    w1, b1 = take(16, 10240), take(16)
    w2, b2 = take(2, 16), take(2)
    logits = F.linear(F.relu(F.linear(x, w1, b1)), w2, b2)
    if not train:
        return torch.softmax(logits, 1)[:, 1]
    loss = F.cross_entropy(logits, lab.long())
    loss.backward()
    return p.grad, loss.detach()


def exact(case, seed):
    kind = case["kind"]
    if kind == "dedisp":
        y = exact_dedisp(case, seed)
        return None if y is None else dict(status=None, series=y)
    if kind == "classify":
        with torch.no_grad():
            return exact_network(case, seed, False)
    if kind == "gradients":
        return exact_network(case, seed, True)
    return None  # the search's statistics are medians and merged lists: no plain 64-bit form
