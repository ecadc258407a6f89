"""The work a user of this package has it do, as timed cases.

Three families, each through the package's public entry points:

``search``  ``AccelSearch.search`` / ``search_block`` over dedispersed series
            (the per-DM acceleration search, the package's main call);
``trial``   one acceleration trial through the operator classes of
            ``peasoup_b200.transforms``, in the order of the reference's loop
            (resample, R2C, interbin, normalise, harmonic sums, peaks);
``dm``      the per-DM work before the trials through the same classes
            (baseline, padding, R2C, running median, deredden, zap,
            statistics, C2R);
``dedisp``  ``Dedisperser.execute`` over SIGPROC sample rows.

``listed()`` gives the named cases, ``draw(rng)`` one more of the same
ranges; ``prepare`` makes the inputs and the handles a program keeps,
``run`` is one pass, ``work`` what a pass cannot do without and ``exact``
the same results in 64-bit arithmetic from torch and numpy alone.
"""
import math
import os
import tempfile

import numpy as np
import torch

from peasoup_b200 import search, sigproc, transforms
from peasoup_b200.dedisperse import Dedisperser

C_LIGHT = 299792458.0
# the header values of the reference's example filterbank: a 64-channel
# L-band receiver; centre frequency and channel width in Hz
FCH1, FOFF = 1510.0, -1.09
CFREQ_HZ, CH_BW_HZ = 1475.12e6, 1.09e6
TOL, MAX_HARM, MIN_GAP, MIN_FREQ, MAX_FREQ = 1e-4, 16.0, 30, 0.1, 1100.0
B5, B25 = 0.05, 0.5


# ------------------------------------------------------------------- cases
def listed():
    return [
        # the example data's search: 2-bit tutorial file, 2^17 points, one DM
        # trial given as the host array a reader returns; latency and launches
        dict(name="search_2p17_host", kind="search", n=1 << 17, nsamps=131072, ndm=1,
             tsamp=320e-6, acc=50.0, dm_step=2.0, folds=4, min_snr=9.0, birdies=0, host=True,
             per_dm=True, red=False, batch=0, shape=0, plain=False),
        # a zero-acceleration periodicity search of many short DM trials, the
        # series a little longer than the transform
        dict(name="block_2p19_zero_acc", kind="search", n=1 << 19, nsamps=560001, ndm=48,
             tsamp=64e-6, acc=0.0, dm_step=1.0, folds=4, min_snr=7.0, birdies=0, host=False,
             per_dm=True, red=False, batch=0, shape=0, plain=False),
        # a served request's 3*2^k length: padded series from host memory,
        # every trial's own list
        dict(name="block_3x2p19_padded", kind="search", n=3 << 19, nsamps=1500001, ndm=8,
             tsamp=64e-6, acc=150.0, dm_step=5.0, folds=3, min_snr=7.0, birdies=0, host=True,
             per_dm=False, red=False, batch=0, shape=0, plain=False),
        # a wide DM grid with few accelerations per DM trial
        dict(name="block_2p22_few_acc", kind="search", n=1 << 22, nsamps=1 << 22, ndm=24,
             tsamp=64e-6, acc=50.0, dm_step=20.0, folds=4, min_snr=7.0, birdies=0, host=False,
             per_dm=True, red=False, batch=16, shape=6, plain=False),
        # the survey workload (the headline benchmark's shape): red noise,
        # birdies, over a hundred accelerations per DM trial
        dict(name="survey_2p23", kind="search", n=1 << 23, nsamps=1 << 23, ndm=4, tsamp=76e-6,
             acc=100.0, dm_step=0.5, folds=5, min_snr=9.0, birdies=20, host=False, per_dm=True,
             red=True, batch=96, shape=6, plain=False),
        # a long observation in one transform
        dict(name="long_2p26", kind="search", n=1 << 26, nsamps=(1 << 26) - 12345, ndm=1,
             tsamp=64e-6, acc=0.12, dm_step=0.0, folds=5, min_snr=9.0, birdies=0, host=False,
             per_dm=True, red=False, batch=0, shape=0, plain=False),
        # one acceleration trial through the drop-in classes, example-data
        # size: what a program written against the operator API runs
        dict(name="trial_2p17", kind="trial", n=1 << 17, tsamp=320e-6, acc=25.0, folds=4,
             min_snr=9.0),
        # the same at an ordinary survey length
        dict(name="trial_2p22", kind="trial", n=1 << 22, tsamp=64e-6, acc=-37.5, folds=5,
             min_snr=7.0),
        # the per-DM operators of a survey DM trial, padded
        dict(name="dm_2p21", kind="dm", n=1 << 21, nsamps=2000003, tsamp=64e-6, birdies=20),
        # the example filterbank: 64 channels of 2 bits, generated DM list
        dict(name="dedisp_2bit_64ch", kind="dedisp", nsamps=187520, nchans=64, nbits=2,
             tsamp=320e-6, ndm=0, dm_lo=0.0, dm_hi=120.0, killed=0, raw=False, host=True),
        # a 1024-channel 4-bit survey beam
        dict(name="dedisp_4bit_1024ch", kind="dedisp", nsamps=400000, nchans=1024, nbits=4,
             tsamp=64e-6, ndm=100, dm_lo=0.0, dm_hi=300.0, killed=11, raw=False, host=False),
        # the headline block's producer: 8-bit rows to 256 DM trials
        dict(name="dedisp_8bit_64ch", kind="dedisp", nsamps=1 << 22, nchans=64, nbits=8,
             tsamp=76e-6, ndm=256, dm_lo=0.0, dm_hi=127.5, killed=0, raw=False, host=False),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["search", "search", "trial", "dm", "dedisp", "dedisp"])
    if kind == "search":
        n = rng.choice([1 << rng.randint(15, 23), 3 << rng.randint(14, 21)])
        tsamp = rng.choice([64e-6, 76e-6, 128e-6, 256e-6])
        # one to a hundred or so trials per DM trial, 2^31 points in all
        acc = 0.0 if rng.random() < 0.2 else 0.5 * _log(rng, 1.5, 100.0) * _acc_step(n, tsamp)
        per = max(1.0, 2.0 * acc / _acc_step(n, tsamp) + 3.0)
        ndm = max(1, min(int(_log(rng, 1, 64)), int((1 << 31) / (n * per)), (1 << 27) // n))
        return dict(kind=kind, n=n, nsamps=int(n * rng.uniform(0.85, 1.2)), ndm=ndm, tsamp=tsamp,
                    acc=acc, dm_step=rng.uniform(0.2, 10.0), folds=rng.randint(1, 5),
                    min_snr=rng.choice([7.0, 9.0]), birdies=rng.choice([0, 0, 20]),
                    host=rng.random() < 0.3, per_dm=rng.random() < 0.7, red=rng.random() < 0.3,
                    batch=0, shape=0, plain=rng.random() < 0.15)
    if kind == "trial":
        n = rng.choice([1, 3]) << rng.randint(14, 22)
        return dict(kind=kind, n=n, tsamp=rng.choice([64e-6, 128e-6, 320e-6]),
                    acc=rng.uniform(-100.0, 100.0), folds=rng.randint(1, 5),
                    min_snr=rng.choice([7.0, 9.0]))
    if kind == "dm":
        n = rng.choice([1, 3]) << rng.randint(15, 22)
        return dict(kind=kind, n=n, nsamps=int(n * rng.uniform(0.8, 1.0)),
                    tsamp=rng.choice([64e-6, 128e-6, 320e-6]), birdies=rng.choice([0, 20]))
    nbits = rng.choice([1, 2, 4, 8, 8, 16])
    nchans = 8 * int(_log(rng, 2, 512))
    ndm = int(_log(rng, 5, 300))
    host = rng.random() < 0.3
    most = min(5e10 / (ndm * nchans), (1 << 28) * 8.0 / (nchans * nbits), 3e9 / (4 * ndm),
               (1 << 28) / nchans, 4e6)
    return dict(kind=kind, nsamps=20000 + int(_log(rng, 5e3, max(1e4, most))), nchans=nchans,
                nbits=nbits, tsamp=rng.choice([64e-6, 128e-6, 320e-6]), ndm=ndm,
                dm_lo=rng.choice([0.0, 20.0]), dm_hi=_log(rng, 30.0, 150.0),
                killed=rng.choice([0, 0, nchans // 10]), raw=rng.random() < 0.3, host=host)


# ------------------------------------------------------------------ inputs
def _series(ndm, nsamps, tsamp, seed, acc, red, n):
    """Dedispersed series as the search meets them: white noise (8-bit
    quantised with red noise in the survey form) and an accelerated pulsar
    that is strongest in the middle DM trial."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 13)
    rng = np.random.default_rng([int(seed), n])
    out = torch.empty((ndm, (nsamps + 3) // 4 * 4), dtype=torch.float32, device="cuda")
    i = torch.arange(nsamps, device="cuda", dtype=torch.float64)
    # slow enough for several harmonics below the search's 1100 Hz, fast
    # enough that the shortest series hold a few hundred turns
    period = float(rng.uniform(0.02, 0.08)) if n * tsamp > 30 else float(rng.uniform(0.005, 0.02))
    k = float(rng.uniform(-0.9, 0.9)) * acc * tsamp / (2.0 * C_LIGHT)
    phi = (i - k * i * (i - n)) * (tsamp / period)
    sig = 0.05 / 2.3548
    pulse = torch.exp(-0.5 * ((phi - torch.round(phi)) / sig) ** 2).float()
    del i, phi
    # about 25 sigma folded: its harmonics well above threshold
    amp = 25.0 / math.sqrt(nsamps * 0.05)
    if red:  # 1/f^1.5 noise below 1 Hz
        z = torch.zeros(nsamps // 2 + 1, dtype=torch.complex64, device="cuda")
        m = min(z.numel(), int(nsamps * tsamp) + 1)
        f = torch.arange(1, m, device="cuda", dtype=torch.float64) / (nsamps * tsamp)
        a = (f ** -0.75 * math.sqrt(nsamps / 2.0)).float()
    for d in range(ndm):
        x = torch.randn(nsamps, generator=g, device="cuda")
        x += pulse * (amp * math.exp(-abs(d - ndm // 2)))
        if red:
            w = torch.randn((m - 1, 2), generator=g, device="cuda")
            z[1:m] = torch.view_as_complex(w) * a
            x += torch.fft.irfft(z, n=nsamps)
            x = torch.clamp(torch.round(128.0 + 20.0 * x), 0.0, 255.0)
        out[d, :nsamps] = x
    return out


def _birdies(count, seed):
    rng = np.random.default_rng([int(seed), 5])
    return (np.sort(rng.uniform(1.0, 1000.0, count)).astype(np.float32),
            np.full(count, 0.1, np.float32))


def _dms(c):
    return (np.float32(c["dm_step"]) * np.arange(c["ndm"], dtype=np.float32)).astype(np.float32)


def _samples(c, seed):
    """(nsamps, nchans) sample values in mid-range noise, and the packed rows."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 31 + 7)
    top = (1 << c["nbits"]) - 1
    ns, nc, b = c["nsamps"], c["nchans"], c["nbits"]
    v = torch.empty((ns, nc), dtype=torch.uint8 if b <= 8 else torch.int32, device="cuda")
    for r in range(0, ns, 1 << 16):
        e = min(ns, r + (1 << 16))
        x = torch.randn((e - r, nc), generator=g, device="cuda")
        v[r:e] = torch.clamp(torch.round(top / 2.0 + max(0.5, (top + 1) / 6.0) * x), 0, top).to(v.dtype)
    if b == 8:
        return v, v
    if b == 16:
        return v, torch.stack([(v & 255), (v >> 8)], 2).to(torch.uint8).reshape(ns, 2 * nc)
    per = 8 // b
    w = v.reshape(ns, nc // per, per)
    rows = torch.zeros((ns, nc // per), dtype=torch.uint8, device="cuda")
    for k in range(per):
        rows |= w[:, :, k] << (k * b)
    return v, rows


def _dm_list(c):
    return np.linspace(c["dm_lo"], c["dm_hi"], c["ndm"]).astype(np.float32)


def _foff(c):
    return FOFF * 64.0 / c["nchans"] if c["nchans"] > 64 else FOFF


def _kill(c):
    k = np.ones(c["nchans"], np.int32)
    if c["killed"]:
        k[np.random.default_rng(c["nchans"]).choice(c["nchans"], c["killed"], False)] = 0
    return k


def _filterbank(c):
    """The filterbank a program opened: its header (the rows are in hand)."""
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "beam.fil")
        sigproc.write_header(path, sigproc.make_header(
            source_name="beam", tsamp=c["tsamp"], fch1=FCH1, foff=_foff(c), nchans=c["nchans"],
            nbits=c["nbits"], nifs=1, nsamples=c["nsamps"]))
        return sigproc.SigprocFilterbank(path, 0, c["nsamps"])


# ----------------------------------------------------------- prepare / run
ROWS = 4096  # of the candidate table that a program keeps


def _table(fields):
    return dict({k: np.zeros(ROWS, np.float32 if k in ("snr", "freq", "acc", "dm") else np.int32)
                 for k in fields}, count=0)


def _tabulate(table, columns):
    """Writes the pass's candidates to the program's table, whose rows past
    the last one stay zero."""
    n, old = min(ROWS, len(next(iter(columns.values())))), min(ROWS, table["count"])
    for k, v in columns.items():
        table[k][:n] = v[:n]
        if old > n:
            table[k][n:old] = 0
    table["count"] = len(next(iter(columns.values())))
    return {k: v.copy() if isinstance(v, np.ndarray) else v for k, v in table.items()}


def prepare(case, seed):
    c = case
    s = {"case": c}
    if c["kind"] == "search":
        block = _series(c["ndm"], c["nsamps"], c["tsamp"], seed, c["acc"], c["red"], c["n"])
        rows = block[:, :c["nsamps"]]
        s["series"] = (np.ascontiguousarray(rows.cpu().numpy()) if c["host"]
                       else [rows[d] for d in range(c["ndm"])])
        s["dms"] = _dms(c)
        s["table"] = _table(("snr", "freq", "acc", "dm", "nh", "dm_idx", "nassoc", "trial",
                             "dm_pos"))
        bf, bw = _birdies(c["birdies"], seed)
        s["search"] = search.AccelSearch(search.SearchParams(
            fft_size=c["n"], tsamp=c["tsamp"], acc_lo=-c["acc"], acc_hi=c["acc"],
            nharmonics=c["folds"], min_snr=c["min_snr"], cfreq_hz=CFREQ_HZ, ch_bw_hz=CH_BW_HZ,
            birdie_freqs=bf, birdie_widths=bw, batch=c["batch"], harm_shape=c["shape"],
            mode="plain" if c["plain"] else "batched"))
    elif c["kind"] == "trial":
        n, b = c["n"], c["n"] // 2 + 1
        x = _series(1, n, c["tsamp"], seed, 0.0, False, n)[0, :n].contiguous()
        s["tim"] = transforms.DeviceTimeSeries(n, c["tsamp"], x)
        s["tim_r"] = transforms.DeviceTimeSeries(n, c["tsamp"])
        s["fs"] = transforms.DeviceFourierSeries(b, _bin_width(n, c["tsamp"]))
        s["ps"] = transforms.DevicePowerSpectrum(s["fs"])
        s["sums"] = transforms.HarmonicSums(s["ps"], c["folds"])
        s["resampler"] = transforms.TimeDomainResampler()
        s["r2c"] = transforms.CuFFTerR2C(n)
        s["former"] = transforms.SpectrumFormer()
        # white unit-variance noise: the interbinned amplitude's statistics
        s["norm"] = transforms.SpectrumNormaliser(1.15 / math.sqrt(n), 0.45 / math.sqrt(n), n)
        s["folder"] = transforms.HarmonicFolder(s["sums"])
        s["finder"] = transforms.PeakFinder(c["min_snr"], MIN_FREQ, MAX_FREQ, b)
        s["table"] = _table(("snr", "freq", "nh"))
        s["distiller"] = transforms.HarmonicDistiller(TOL, MAX_HARM, False)
    elif c["kind"] == "dm":
        n, b = c["n"], c["n"] // 2 + 1
        s["raw"] = _series(1, c["nsamps"], c["tsamp"], seed, 0.0, True, n)[0, :c["nsamps"]]
        s["tim"] = transforms.DeviceTimeSeries(n, c["tsamp"])
        s["fs"] = transforms.DeviceFourierSeries(b, _bin_width(n, c["tsamp"]))
        s["ps"] = transforms.DevicePowerSpectrum(s["fs"])
        s["r2c"], s["c2r"] = transforms.CuFFTerR2C(n), transforms.CuFFTerC2R(n)
        s["former"] = transforms.SpectrumFormer()
        s["dered"] = transforms.Dereddener(b)
        s["zapper"] = transforms.Zapper.from_arrays(*_birdies(c["birdies"], seed))
    else:
        _, rows = _samples(c, seed)
        s["rows"] = rows.cpu().pin_memory() if c["host"] else rows
        dd = Dedisperser(_filterbank(c))
        if c["ndm"]:
            dd.set_dm_list(_dm_list(c))
        else:
            dd.generate_dm_list(c["dm_lo"], c["dm_hi"], 64.0, 1.11)
        if c["killed"]:
            dd.set_killmask(_kill(c))
        s["dd"] = dd
        s["nout"] = c["nsamps"] - dd.get_max_delay()
        s["out"] = torch.empty((len(dd.get_dm_list()), (s["nout"] + 3) // 4 * 4),
                               dtype=torch.float32, device="cuda")
    return s


def run(state):
    s = state
    c = s["case"]
    if c["kind"] == "search":
        if c["ndm"] == 1:
            cand, na, tr = s["search"].search(s["series"][0], float(s["dms"][0]), 0,
                                              per_dm=c["per_dm"])
            pos = np.zeros(len(cand), np.int32)
        else:
            cand, na, tr, pos = s["search"].search_block(s["series"], s["dms"], None,
                                                         per_dm=c["per_dm"])
        out = {k: cand[k] for k in ("snr", "freq", "acc", "dm", "nh", "dm_idx")}
        return _tabulate(s["table"], dict(out, nassoc=na, trial=tr, dm_pos=pos))
    if c["kind"] == "trial":
        s["resampler"].resampleII(s["tim"], s["tim_r"], c["n"], c["acc"])
        s["r2c"].execute(s["tim_r"], s["fs"])
        s["former"].form_interpolated(s["fs"], s["ps"])
        s["norm"].normalise(s["ps"])
        s["folder"].fold(s["ps"])
        cands = transforms.SpectrumCandidates(0.0, 0, c["acc"])
        s["finder"].find_candidates(s["ps"], cands)
        s["finder"].find_candidates(s["sums"], cands)
        kept = s["distiller"].distill(cands.cands)
        return {"spectrum": s["ps"].data, "sums": [h.data for h in s["sums"].folds],
                "cands": _tabulate(s["table"], {k: [getattr(q, k) for q in kept]
                                                for k in ("snr", "freq", "nh")})}
    if c["kind"] == "dm":
        tim, fs, ps = s["tim"], s["fs"], s["ps"]
        tim.data[:c["nsamps"]].copy_(s["raw"])
        passes = tim.remove_baseline(c["nsamps"])
        tim.fill(c["nsamps"], c["n"], 0.0)
        s["r2c"].execute(tim, fs)
        s["former"].form(fs, ps)
        s["dered"].calculate_median(ps)
        s["dered"].deredden(fs)
        s["zapper"].zap(fs)
        s["former"].form_interpolated(fs, ps)
        mean, rms, std = transforms.stats.stats(ps.data, ps.get_nbins())
        s["c2r"].execute(fs, tim)
        return {"series": tim.data, "median": s["dered"].median, "passes": passes,
                "stats": np.array([mean, rms, std], np.float32)}
    s["dd"].execute(s["rows"], c["nsamps"], s["out"], raw=c["raw"])
    return s["out"][:, :s["nout"]]


# -------------------------------------------------------------------- work
def _fft_flops(n):
    return 2.5 * n * math.log2(n)


def _trial_flops(n, folds):
    return _fft_flops(n) + n / 2 * ((1 << folds) - 1 + folds + 12)


def work(case):
    c = case
    if c["kind"] == "search":
        ntr = sum(len(_acc_list(c, float(d))) for d in _dms(c))
        # each series read once; per trial its resampled series read and its
        # spectrum handed from the transform to the harmonic sums (12 n bytes,
        # the roofline of the fused search), per DM trial 24 n for the rest
        return {"bytes": 12.0 * c["n"] * ntr + 24.0 * c["n"] * c["ndm"],
                "flops": ntr * _trial_flops(c["n"], c["folds"]) + c["ndm"] * 2 * _fft_flops(c["n"])}
    if c["kind"] == "trial":
        # the operators are calls of their own: each reads its input and writes its output once
        n, b = c["n"], c["n"] // 2 + 1
        by = 8 * n + (4 * n + 8 * b) + 12 * b + 8 * b + 4 * b * (1 + c["folds"]) * 2
        return {"bytes": float(by), "flops": _trial_flops(n, c["folds"])}
    if c["kind"] == "dm":
        n, b, m = c["n"], c["n"] // 2 + 1, c["nsamps"]
        by = 8 * m + 8 * m + 4 * (n - m) + (4 * n + 8 * b) + 12 * b + 8 * b + 20 * b + 12 * b \
            + 4 * b + (8 * b + 4 * n)
        return {"bytes": float(by), "flops": 2 * _fft_flops(n) + 40.0 * b}
    delays = _delays(c)
    dms = _dm_list(c) if c["ndm"] else _generated(c)
    nout = c["nsamps"] - int(math.floor(float(np.float32(dms.max()) * delays[-1]) + 0.5))
    return {"bytes": c["nsamps"] * c["nchans"] * c["nbits"] / 8.0 + 4.0 * len(dms) * nout,
            "flops": float(len(dms)) * nout * (c["nchans"] - c["killed"])}


# ------------------------------------------- the same in 64-bit arithmetic
def _bin_width(n, tsamp):
    return float(np.float32(1.0 / float(np.float32(np.float32(n) * np.float32(tsamp)))))


def _acc_step(n, tsamp, ddm=0.0):
    f32 = np.float32
    bw = f32(CH_BW_HZ)
    ftop = f32(float(f32(CFREQ_HZ) + bw / f32(2)) / 1e9)
    fbot = f32(float(f32(CFREQ_HZ) - bw / f32(2)) / 1e9)
    inv = f32(1) / (fbot * fbot) - f32(1) / (ftop * ftop)
    tdm = f32(4.15e-3 * float(inv) * float(abs(f32(ddm))))
    pw, ts = f32(64e-6), f32(tsamp)
    broad = f32(math.sqrt(float(tdm * tdm + pw * pw + ts * ts)))
    factor = f32(math.sqrt(float(f32(1.10) * f32(1.10)) - 1.0))
    tobs = f32(n) * ts
    return float(f32(2.0 * float(broad) * 24.0 * C_LIGHT / float(tobs * tobs) * float(factor)))


def _acc_list(c, dm):
    lo, hi = np.float32(-c["acc"]), np.float32(c["acc"])
    if lo == hi:
        return np.array([hi], np.float32)
    step, a, out = np.float32(_acc_step(c["n"], c["tsamp"], dm)), lo, [np.float32(0), hi]
    while a <= hi:
        out.append(a)
        a = np.float32(a + step)
    return np.unique(np.array(out, np.float32))


def _interbin(x):
    prev = torch.cat([torch.zeros_like(x[:1]), x[:-1]])
    return torch.sqrt(torch.maximum(x.abs() ** 2, 0.5 * (x - prev).abs() ** 2))


def _scrunch(a):
    m = a.numel() // 5
    return a[:5 * m].reshape(m, 5).median(1).values


def _stretch(a, count):
    step = torch.tensor(np.float32(a.numel() - 1) / np.float32(count - 1), device=a.device)
    x = torch.arange(count, device=a.device).to(torch.float32) * step
    j = x.long().clamp(max=a.numel() - 1)
    w = (x - j.to(torch.float32)).double()
    hi = a[(j + 1).clamp(max=a.numel() - 1)]
    return a[j] + torch.where(w > 1e-5, w * (hi - a[j]), torch.zeros_like(w))


def _median(amp, bw):
    n = amp.numel()
    m5 = _scrunch(amp)
    m25 = _scrunch(m5)
    m125 = _scrunch(m25)
    p5 = min(n, int(float(np.float32(B5)) / bw))
    p25 = max(p5, min(n, int(float(np.float32(B25)) / bw)))
    out = _stretch(m125, n)
    out[:p25] = _stretch(m25, n)[:p25]
    out[:p5] = _stretch(m5, n)[:p5]
    return out


def _dm_stage(x, c, birdies):
    """Dereddened series, median and (mean, rms, std) of one DM trial."""
    n, bw = c["n"], _bin_width(c["n"], c["tsamp"])
    x = x[:n].double()
    t = torch.zeros(n, dtype=torch.float64, device=x.device)
    t[:x.numel()] = x - x.mean()
    f = torch.fft.rfft(t)
    med = _median(f.abs(), bw)
    f /= med
    f[:5] = 0
    w32 = np.float32(bw)
    for fr, wd in zip(*birdies):
        lo = max(0, int(math.floor(float(np.float32(fr - wd) / w32))))
        hi = min(f.numel() - 1, int(math.ceil(float(np.float32(fr + wd) / w32))))
        if lo < f.numel():
            f[lo:hi] = 1
    p = _interbin(f)
    mean, rms = float(p.mean()), math.sqrt(float((p * p).mean()))
    return torch.fft.irfft(f, n=n) * n, med, (mean, rms, math.sqrt(rms * rms - mean * mean))


def _resampled(x, n, acc, tsamp):
    k = float(np.float32(np.float32(acc) * np.float32(tsamp))) / (2 * C_LIGHT)
    i = torch.arange(n, device=x.device, dtype=torch.float64)
    j = torch.round(i + i * k * (i - n)).long()
    return torch.where((j >= 0) & (j < n), x[j.clamp(0, n - 1)], torch.zeros_like(x[:1]))


def _sums(p, folds):
    i = torch.arange(p.numel(), device=p.device)
    val, out = p.clone(), []
    for h in range(1, folds + 1):
        for m in range(1, 1 << h, 2):
            val += p[(i * m + (1 << (h - 1))) >> h]
        out.append(val / math.sqrt(2.0 ** h))
    return out


def _peaks(spec, h, bw, thresh, per):
    """(bin, value, frequency) of each cluster over the threshold."""
    size = spec.numel()
    nyq = float(np.float32(bw * size))
    orig = np.float32(2.0 * (size - 1.0))
    start = int(float(orig * (np.float32(MIN_FREQ) / np.float32(nyq))) * 2.0 ** h)
    end = min(size, int(float(np.float32(MAX_FREQ)) / bw * 2.0 ** h))
    fac = 1.0 / size * nyq / 2.0 ** h
    idx = torch.nonzero(spec[start:end] > thresh).reshape(-1) + start
    val = spec[idx].cpu().numpy()
    idx = idx.cpu().numpy()
    k = 0
    while k < len(idx):
        at, best, last = idx[k], val[k], idx[k]
        k += 1
        while k < len(idx) and idx[k] - last < MIN_GAP:
            if val[k] > best:
                at, best, last = idx[k], val[k], idx[k]
            k += 1
        per.append((float(best), float(at) * fac, h))


def _harmonic_distilled(cands):
    """Survivors in order of S/N; (snr, freq, nh, ...) tuples."""
    cands = sorted(cands, key=lambda q: -q[0])
    if not cands:
        return []
    up, dn = 1.0 + TOL, 1.0 - TOL
    alive = np.ones(len(cands), bool)
    freq = np.array([q[1] for q in cands])
    nh = np.array([q[2] for q in cands])
    jj = np.arange(1, int(MAX_HARM) + 1)[None, :, None]
    kk = np.arange(1, 2 ** int(nh.max()) + 1)[None, None, :]
    for i in range(len(cands)):
        if not alive[i]:
            continue
        f, den = freq[i + 1:, None, None], (2 ** nh[i + 1:])[:, None, None]
        r = kk * f / (jj * freq[i])
        alive[i + 1:] &= ~((r > dn) & (r < up) & (kk <= den)).any((1, 2))
    return [q for q, a in zip(cands, alive) if a]


def _accel_distilled(cands, tobs):
    cands = sorted(cands, key=lambda q: -q[0])
    alive = [True] * len(cands)
    for i, q in enumerate(cands):
        if not alive[i]:
            continue
        edge = q[1] * TOL
        for j in range(i + 1, len(cands)):
            r = cands[j]
            af = q[1] + (q[3] - r[3]) * q[1] * tobs / C_LIGHT
            if (q[1] - edge < r[1] < af + edge) if af > q[1] else (af - edge < r[1] < q[1] + edge):
                alive[j] = False
    return [q for q, a in zip(cands, alive) if a]


def _exact_search(c, seed):
    block = _series(c["ndm"], c["nsamps"], c["tsamp"], seed, c["acc"], c["red"], c["n"])
    bw = _bin_width(c["n"], c["tsamp"])
    out = []
    for d, dm in enumerate(_dms(c)):
        x, _, (mean, _, std) = _dm_stage(block[d, :c["nsamps"]], c, _birdies(c["birdies"], seed))
        per = []
        for acc in _acc_list(c, float(dm)):
            f = torch.fft.rfft(_resampled(x, c["n"], acc, c["tsamp"]))
            p = (_interbin(f) - mean * c["n"]) / (std * c["n"])
            del f
            found = []
            for h, sp in enumerate([p] + _sums(p, c["folds"])):
                _peaks(sp, h, bw, c["min_snr"], found)
            per += [q + (float(acc), float(dm)) for q in _harmonic_distilled(found)]
        out += _accel_distilled(per, float(np.float32(c["n"]) * np.float32(c["tsamp"]))) \
            if c["per_dm"] else per
    return _exact_table(out, {"snr": 0, "freq": 1, "acc": 3, "dm": 4},
                        ("nh", "dm_idx", "nassoc", "trial", "dm_pos", "count"))


def _exact_table(cands, columns, rest):
    r = dict.fromkeys(rest)
    for k, at in columns.items():
        r[k] = np.zeros(ROWS, np.float64)
        r[k][:len(cands)] = [q[at] for q in cands[:ROWS]]
    return r


def _delays(c):
    f32 = np.float32
    out = []
    for k in range(c["nchans"]):
        a, b = f32(1) / (f32(FCH1) + f32(k) * f32(_foff(c))), f32(1) / f32(FCH1)
        out.append(f32(4.15e3 / float(f32(c["tsamp"])) * float(a * a - b * b)))
    return np.array(out, np.float32)


def _generated(c):
    """The DM list whose steps keep the smearing within a tolerance of 1.11."""
    ts, tol, width = float(np.float32(c["tsamp"])) * 1e6, float(np.float32(1.11)), 64.0
    f = (FCH1 + (c["nchans"] // 2 - 0.5) * float(np.float32(_foff(c)))) * 1e-3
    a2 = (8.3 * float(np.float32(_foff(c))) / f ** 3) ** 2
    b2 = a2 * (c["nchans"] ** 2 / 16.0)
    k0 = (ts * ts + width * width) * (tol * tol - 1.0)
    dms = [np.float32(c["dm_lo"])]
    while dms[-1] < np.float32(c["dm_hi"]):
        p = float(dms[-1])
        k = k0 + tol * tol * a2 * p * p
        dms.append(np.float32((b2 * p + math.sqrt(-a2 * b2 * p * p + (a2 + b2) * k)) / (a2 + b2)))
    return np.array(dms, np.float32)


def _exact_dedisp(c, seed):
    v, _ = _samples(c, seed)
    v = v.t().contiguous()
    dms = _dm_list(c) if c["ndm"] else _generated(c)
    delays = _delays(c)
    shift = np.rint(dms[:, None] * delays[None, :]).astype(np.int64)
    nout = c["nsamps"] - int(math.floor(float(dms.max() * delays[-1]) + 0.5))
    live = np.flatnonzero(_kill(c))
    top = (1 << c["nbits"]) - 1
    out = torch.empty((len(dms), nout), dtype=torch.float64, device="cuda")
    acc = torch.empty(nout, dtype=torch.int32, device="cuda")
    for d in range(len(dms)):
        acc.zero_()
        for ch in live:
            acc += v[ch, shift[d, ch]:shift[d, ch] + nout]
        out[d] = acc
    if not c["raw"]:
        out.sub_(0.5 * c["nchans"] * top).mul_(1.0 / (top * math.sqrt(c["nchans"]))).add_(0.5)
    return out


def exact(case, seed):
    c = case
    if c["kind"] == "search":
        # the harmonic sums in 64 bits over the largest blocks take too long
        points = c["n"] * sum(len(_acc_list(c, float(d))) for d in _dms(c))
        return None if points > 1 << 33 else _exact_search(c, seed)
    if c["kind"] == "trial":
        n = c["n"]
        x = _series(1, n, c["tsamp"], seed, 0.0, False, n)[0, :n].double()
        p = _interbin(torch.fft.rfft(_resampled(x, n, c["acc"], c["tsamp"])))
        f32 = np.float32
        mean, std = f32(f32(1.15 / math.sqrt(n)) * f32(n)), f32(f32(0.45 / math.sqrt(n)) * f32(n))
        p = (p - float(mean)) / float(std)
        sums, found = _sums(p, c["folds"]), []
        for h, sp in enumerate([p] + sums):
            _peaks(sp, h, _bin_width(n, c["tsamp"]), c["min_snr"], found)
        kept = _harmonic_distilled(found)
        return {"spectrum": p, "sums": sums,
                "cands": _exact_table(kept, {"snr": 0, "freq": 1}, ("nh", "count"))}
    if c["kind"] == "dm":
        x = _series(1, c["nsamps"], c["tsamp"], seed, 0.0, True, c["n"])[0, :c["nsamps"]]
        t, med, st = _dm_stage(x, c, _birdies(c["birdies"], seed))
        return {"series": t, "median": med, "passes": None, "stats": np.array(st)}
    return _exact_dedisp(c, seed)
