"""Timed cases of the generalized Lomb-Scargle and adjoint-NFFT paths.

Every case is a call that a user of the package makes: the reference-style
Python processes (host arrays in, host arrays out) or the C entry points of
libcuvgls through their bindings (device buffers in and out, as a pipeline
that keeps its data on the GPU calls them).  Light curves follow the
benchmark's: irregular sorted times, a sinusoid plus noise, heteroscedastic
errors, frequencies (k0 + k) / (spp T).

  listed()            the cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) inputs on the GPU (host arrays for the host entry points)
  run(state)          one call, its outputs
  work(case)          bytes and operations the call cannot do without
  exact(case, seed)   the outputs in 64 bits, from plain torch

Handles and processes are kept by this module, one per (window, sigma, m), as
a program that processes many batches keeps them.
"""
import ctypes
import math

import numpy as np
import torch

from cuvarbase_gb300 import _lib
from cuvarbase_gb300.cunfft import NFFTAsyncProcess
from cuvarbase_gb300.lombscargle import LombScargleAsyncProcess, lomb_scargle_direct_sums

AUTO = -1.0  # sigma below zero: the library picks window, sigma and m

MODES = {"standard": _lib.MODE_STANDARD, "floating": _lib.MODE_FLOATING_MEAN,
         "window": _lib.MODE_WINDOW}


def listed():
    return [
        # one short light curve, already on the device: a call in a pipeline
        # loop, where launches and their latency are all there is
        dict(name="one_short", kind="raw", curves=1, nmin=211, nmax=211, nf=3000, sigma=AUTO, m=8,
             mode="floating", prior=0.0),
        # the plain use of the reference's API: one curve of 1,000 points over
        # ten years, sigma 2 and m 8, run() + finish()
        dict(name="run_one", kind="run", curves=1, nmin=1000, nmax=1000, nf=50000, sigma=2.0, m=8,
             mode="floating", prior=0.0),
        # a captured plan of a fixed-shape batch, replayed as data arrives
        dict(name="plan_16", kind="plan", curves=16, nmin=50, nmax=5000, nf=20000, sigma=AUTO, m=8,
             mode="floating", prior=0.0),
        # a batch of the serving loop: every request has its own point count
        # and its own number of frequencies (10^4 to 10^6), host-prepared
        dict(name="ragged_serve", kind="prepared", curves=48, nmin=100, nmax=20000, nf=10000,
             nfmax=1000000, sigma=AUTO, m=8, mode="floating", prior=0.0),
        # the batched workload of the benchmark, a fifth of its curves
        dict(name="batch_auto", kind="raw", curves=2000, nmin=50, nmax=5000, nf=100000, sigma=AUTO,
             m=8, mode="floating", prior=0.0),
        # the same curves at the reference's defaults, sigma 4 and m 8
        dict(name="batch_sigma4", kind="raw", curves=400, nmin=50, nmax=5000, nf=100000, sigma=4.0,
             m=8, mode="standard", prior=0.0),
        # a survey of short curves of which only the best frequency is kept
        dict(name="survey_best", kind="best", curves=20000, nmin=20, nmax=300, nf=20000, sigma=AUTO,
             m=8, mode="floating", prior=0.0),
        # one dense curve of 10^6 points to 1,000 cycles a day
        dict(name="dense", kind="prepared", curves=1, nmin=1000000, nmax=1000000, nf=18250000,
             nfmax=18250000, sigma=AUTO, m=8, mode="floating", prior=0.0),
        # adjoint NFFTs of a batch, complex output (sigma 2, m 8)
        dict(name="nfft_batch", kind="nfft", curves=1000, nmin=50, nmax=5000, nf=100000, sigma=2.0,
             m=8),
        # the NFFT process with use_double: exact sums, complex128, host to host
        dict(name="nfft_double", kind="nfft64", curves=4, nmin=300, nmax=2000, nf=20000),
        # use_fft=False: the reference's direct-sum kernel
        dict(name="direct_sums", kind="direct", curves=8, nmin=300, nmax=2000, nf=10000,
             mode="floating", prior=0.0),
        # the multi-harmonic model of one curve, host to host in FP64, from
        # two cycles over the time span on (below, the model's harmonics are
        # not independent and its system is close to singular)
        dict(name="harmonics", kind="harmonics", curves=1, nmin=1000, nmax=1000, nf=20000, nharms=3),
    ]


FIRST_HARMONIC_BIN = 10  # frequencies of the multi-harmonic case: (10 + k) / (5 T)


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["raw", "raw", "run", "plan", "prepared", "sigma", "best", "dense", "nfft",
                       "nfft64", "direct", "harmonics"])
    mode = rng.choice(["floating", "floating", "standard", "window"])
    prior = rng.choice([0.0, 0.0, 0.0, 2.0])
    lo = _log_int(rng, 20, 1000)
    hi = lo * rng.choice([1, 2, 5, 20])
    if kind == "raw":
        nf = _log_int(rng, 1000, 300000)
        return dict(kind="raw", curves=_log_int(rng, 1, max(2, min(2000, int(1.5e8 / nf)))), nmin=lo,
                    nmax=min(hi, 5000), nf=nf, sigma=AUTO, m=8, mode=mode, prior=prior)
    if kind == "sigma":
        nf, s = _log_int(rng, 3000, 300000), rng.choice([2.0, 4.0, 5.0])
        return dict(kind="raw", curves=_log_int(rng, 1, max(2, min(1000, int(1.2e8 / (s * nf))))),
                    nmin=lo, nmax=min(hi, 5000), nf=nf, sigma=s, m=8, mode=mode, prior=prior)
    if kind == "run":
        return dict(kind="run", curves=_log_int(rng, 1, 32), nmin=lo, nmax=min(hi, 5000),
                    nf=_log_int(rng, 2000, 100000), sigma=rng.choice([AUTO, 2.0, 4.0]), m=8,
                    mode=mode, prior=prior)
    if kind == "plan":
        return dict(kind="plan", curves=_log_int(rng, 2, 256), nmin=lo, nmax=min(hi, 5000),
                    nf=_log_int(rng, 5000, 50000), sigma=AUTO, m=8, mode=mode, prior=prior)
    if kind == "prepared":
        nf = _log_int(rng, 3000, 50000)
        return dict(kind="prepared", curves=_log_int(rng, 4, 64), nmin=max(lo, 100),
                    nmax=max(lo, 100) * rng.choice([2, 20]), nf=nf,
                    nfmax=nf * rng.choice([2, 10, 20]), sigma=AUTO, m=8, mode=mode, prior=prior)
    if kind == "best":
        nf = _log_int(rng, 5000, 50000)
        return dict(kind="best", curves=_log_int(rng, 500, max(501, min(20000, int(3e8 / nf)))),
                    nmin=rng.randrange(20, 100), nmax=rng.randrange(100, 400), nf=nf, sigma=AUTO,
                    m=8, mode="floating", prior=0.0)
    if kind == "dense":
        n, nf = _log_int(rng, 100000, 1000000), _log_int(rng, 1000000, 18000000)
        return dict(kind="prepared", curves=1, nmin=n, nmax=n, nf=nf, nfmax=nf, sigma=AUTO, m=8,
                    mode=mode, prior=prior)
    if kind == "nfft":
        nf = _log_int(rng, 3000, 200000)
        s = rng.choice([AUTO, 2.0, 4.0])
        return dict(kind="nfft", curves=_log_int(rng, 1, max(2, min(1000, int(5e7 / nf)))), nmin=lo,
                    nmax=min(hi, 5000), nf=nf, sigma=s, m=8)
    n = _log_int(rng, 50, 1500)
    nf = _log_int(rng, 1000, 20000)
    if kind == "harmonics":
        return dict(kind="harmonics", curves=1, nmin=n, nmax=n, nf=nf, nharms=rng.randrange(1, 5))
    few = rng.randrange(1, 6)
    if kind == "nfft64":
        return dict(kind="nfft64", curves=few, nmin=n, nmax=n + rng.randrange(0, 400), nf=nf)
    return dict(kind="direct", curves=few, nmin=n, nmax=n + rng.randrange(0, 400), nf=nf, mode=mode,
                prior=prior)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _batch(case, seed):
    """Host light curves: sorted times over 100 to 3,650 d (1,000 d for the
    survey, 3,650 d for the dense curve), one sinusoid each, noise, errors.
    The sizes of the curves belong to the case, their values to the seed."""
    c = case["curves"]
    rng = np.random.default_rng([c, case["nmin"], case["nmax"], case["nf"]])
    if case["kind"] == "best":
        N = rng.integers(case["nmin"], case["nmax"] + 1, c).astype(np.int64)
    else:
        N = np.round(np.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"]), c)))
        N = N.astype(np.int64)
    nf = np.full(c, case["nf"], np.int64)
    if case.get("nfmax", case["nf"]) > case["nf"]:
        nf = np.round(np.exp(rng.uniform(math.log(case["nf"]), math.log(case["nfmax"]), c)))
        nf = nf.astype(np.int64)
    rng = np.random.default_rng(seed)
    survey, dense = case["kind"] == "best", case["nmin"] >= 100000
    T = np.full(c, 1000.0 if survey else 3650.0) if survey or dense else rng.uniform(100, 3650, c)
    spp = 1.0 if survey else 5.0
    off = np.zeros(c + 1, np.int64)
    off[1:] = np.cumsum(N)
    cid = np.repeat(np.arange(c), N)
    t = np.sort(rng.uniform(0, 1, int(off[-1])) + cid) - cid
    t = np.clip(t, 0.0, 1.0) * T[cid]
    df = 1.0 / (spp * T)
    # the injected frequency lies inside the band
    k_inj = np.maximum(1, (nf * rng.uniform(0.05, 0.95, c)).astype(np.int64))
    amp = rng.uniform(0.2, 0.5, c) if survey else rng.uniform(0.05, 0.5, c)
    sn = np.full(c, 0.1) if survey else rng.uniform(0.02, 0.2, c)
    ph = rng.uniform(0, 2 * np.pi, c)
    y = (amp[cid] * np.sin(2 * np.pi * (k_inj * df)[cid] * t + ph[cid])
         + rng.normal(0, 1, t.size) * sn[cid])
    y += rng.normal(10.0, 1.0, c)[cid]
    dy = np.exp(rng.normal(math.log(0.05), 0.3, t.size))
    return dict(N=N, nf=nf, off=off, cid=cid, t=t, y=y, dy=dy, df=df, T=T, k0=1)


def _prepare_host(b):
    """The reference's host preparation: means removed, normalised weights,
    yw = w (y - ybar) and w as float32, YY in FP64."""
    off, cid, N = b["off"], b["cid"], b["N"]

    def red(a):
        return np.add.reduceat(a, off[:-1])

    t = b["t"] - (red(b["t"]) / N)[cid]
    y = b["y"] - (red(b["y"]) / N)[cid]
    w = b["dy"] ** -2
    w = w / red(w)[cid]
    ybar = red(w * y)
    yw = w * (y - ybar[cid])
    yy = red(w * (y - ybar[cid]) ** 2)
    yw32, w32 = yw.astype(np.float32), w.astype(np.float32)
    return dict(t=t, yw=yw32, w=w32, yw64=yw, w64=w, yy=yy, ybar=ybar,
                yw_sum=red(yw32.astype(np.float64)), w_sum=red(w32.astype(np.float64)))


_CURVE = np.dtype([("pt_off", "<i8"), ("n", "<i8"), ("nf", "<i8"), ("k0", "<i8"), ("df", "<f8"),
                   ("yy", "<f8"), ("ybar", "<f8"), ("yw_sum", "<f8"), ("w_sum", "<f8"),
                   ("out_off", "<i8")])
_RAW = np.dtype([("pt_off", "<i8"), ("n", "<i8"), ("nf", "<i8"), ("k0", "<i8"), ("df", "<f8"),
                 ("out_off", "<i8")])
_NFFT = np.dtype([("pt_off", "<i8"), ("n", "<i8"), ("nf", "<i8"), ("f0", "<f8"), ("df", "<f8"),
                  ("out_off", "<i8")])

_handles, _processes = {}, {}


def _handle(case):
    key = (case.get("sigma", 2.0), case.get("m", 8))
    if key not in _handles:
        _handles[key] = _lib.Handle(sigma=key[0], m=key[1])
    return _handles[key]


def _process(case):
    if case["kind"] == "nfft64":
        key = "nfft64"
        if key not in _processes:
            _processes[key] = NFFTAsyncProcess(use_double=True)
    else:
        key = (case["sigma"], case["m"])
        if key not in _processes:
            _processes[key] = LombScargleAsyncProcess(
                sigma="auto" if case["sigma"] < 0 else case["sigma"], m=case["m"])
    return _processes[key]


def _reg(case):
    return float(np.float32(case["prior"] ** -2)) if case.get("prior") else 0.0


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


class _Plan:
    """A captured plan and the buffers that it reads and writes."""

    def __init__(self, handle, inp, out):
        self.ptr, self.out, self.lib = ctypes.c_void_p(), out, _lib.load()
        handle.check(self.lib.cuvgls_gls_plan_create(handle.ptr, ctypes.byref(inp), out.data_ptr(),
                                                     None, None, ctypes.byref(self.ptr)), "plan")

    def __del__(self):
        if self.ptr:
            self.lib.cuvgls_gls_plan_destroy(self.ptr)
            self.ptr = None


def prepare(case, seed):
    kind = case["kind"]
    b = _batch(case, seed)
    c, npts = case["curves"], int(b["off"][-1])
    s = dict(kind=kind, case=case)
    if kind in ("run", "nfft64"):
        spl = [slice(int(b["off"][i]), int(b["off"][i + 1])) for i in range(c)]
        s["proc"] = _process(case)
        if kind == "run":
            s["data"] = [(b["t"][q], b["y"][q], b["dy"][q]) for q in spl]
            s["freqs"] = [df * (1 + np.arange(int(nf))) for df, nf in zip(b["df"], b["nf"])]
        else:
            s["data"] = [(b["t"][q], b["y"][q], int(nf)) for q, nf in zip(spl, b["nf"])]
        return s
    if kind == "harmonics":
        p = _prepare_host(b)
        s.update(t=p["t"], yw=p["yw64"], w=p["w64"], yy=float(p["yy"][0]),
                 freqs=float(b["df"][0]) * (FIRST_HARMONIC_BIN + np.arange(case["nf"])))
        return s
    out_off = np.zeros(c + 1, np.int64)
    out_off[1:] = np.cumsum(b["nf"])
    tab = np.zeros(c, {"raw": _RAW, "plan": _RAW, "best": _RAW, "nfft": _NFFT}.get(kind, _CURVE))
    tab["pt_off"], tab["n"], tab["nf"], tab["df"] = b["off"][:-1], b["N"], b["nf"], b["df"]
    tab["out_off"] = out_off[:-1]
    nout = int(out_off[-1])
    s["handle"], s["table"] = _handle(case), tab
    if kind == "nfft":
        inp = _lib.NfftInput()
        tab["f0"] = b["df"] * b["k0"]
        s["in"] = [_dev(b["t"]), _dev(b["y"].astype(np.float32))]
        inp.t, inp.y = (x.data_ptr() for x in s["in"])
        s["out"] = torch.empty(nout, dtype=torch.complex64, device="cuda")
    elif kind in ("raw", "plan", "best"):
        inp = _lib.RawInput()
        tab["k0"] = b["k0"]
        s["in"] = [_dev(b["t"]), _dev(b["y"]), _dev(b["dy"])]
        inp.t, inp.y, inp.dy = (x.data_ptr() for x in s["in"])
        if kind == "best":
            s["out"] = (torch.empty(c, dtype=torch.int64, device="cuda"),
                        torch.empty(c, dtype=torch.float32, device="cuda"))
        else:
            s["out"] = torch.empty(nout, dtype=torch.float32, device="cuda")
    else:
        inp = _lib.GlsInput()
        p = _prepare_host(b)
        tab["k0"] = b["k0"]
        for k in ("yy", "ybar", "yw_sum", "w_sum"):
            tab[k] = p[k]
        s["in"] = [_dev(p["t"]), _dev(p["yw"]), _dev(p["w"])]
        inp.t, inp.yw, inp.w = (x.data_ptr() for x in s["in"])
        s["out"] = torch.empty(nout, dtype=torch.float32, device="cuda")
    if kind != "nfft":
        inp.mode = MODES[case["mode"]]
        inp.reg[0] = inp.reg[1] = _reg(case)
    inp.n_curves, inp.curves, inp.flags = c, tab.ctypes.data, 0
    inp.n_points_total, inp.n_out_total = npts, nout
    s["inp"] = inp
    if kind == "plan":
        s["plan"] = _Plan(s["handle"], inp, s["out"])
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "run":
        case, proc = s["case"], s["proc"]
        res = proc.run(s["data"], freqs=s["freqs"], floating_mean=case["mode"] != "standard",
                       window=case["mode"] == "window",
                       amplitude_prior=case["prior"] if case["prior"] else None)
        proc.finish()
        return [p for _, p in res]
    if kind == "nfft64":
        res = s["proc"].run(s["data"], samples_per_peak=5)
        s["proc"].finish()
        return res
    if kind == "harmonics":
        return lomb_scargle_direct_sums(s["t"], s["yw"], s["w"], s["freqs"], s["yy"],
                                        nharms=s["case"]["nharms"])
    lib, h, inp = _lib.load(), s["handle"], s["inp"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "plan":
        _lib.raise_for(lib.cuvgls_gls_plan_launch(s["plan"].ptr, stream), None, "plan launch")
    elif kind == "best":
        k, p = s["out"]
        h.check(lib.cuvgls_gls_raw(h.ptr, ctypes.byref(inp), None, k.data_ptr(), p.data_ptr(),
                                   stream), "best")
    elif kind == "raw":
        h.check(lib.cuvgls_gls_raw(h.ptr, ctypes.byref(inp), s["out"].data_ptr(), None, None,
                                   stream), "raw")
    elif kind == "nfft":
        h.check(lib.cuvgls_nfft_adjoint_batch(h.ptr, ctypes.byref(inp), s["out"].data_ptr(),
                                              stream), "nfft")
    else:
        fn = lib.cuvgls_gls_direct_batch if kind == "direct" else lib.cuvgls_gls_batch
        h.check(fn(h.ptr, ctypes.byref(inp), s["out"].data_ptr(), stream), kind)
    return s["out"]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind, c = case["kind"], case["curves"]

    def mean(lo, hi):  # of a log-uniform number
        return lo if hi <= lo else (hi - lo) / math.log(hi / lo)

    n = mean(case["nmin"], case["nmax"])
    if kind == "best":
        n = 0.5 * (case["nmin"] + case["nmax"])
    nf = mean(case["nf"], case.get("nfmax", case["nf"]))
    per_in = {"raw": 24, "plan": 24, "best": 24, "run": 24, "harmonics": 24, "nfft": 12,
              "nfft64": 16}.get(kind, 16)
    per_out = {"nfft": 8, "nfft64": 16, "harmonics": 8, "best": 0}.get(kind, 4)
    nbytes = c * (n * per_in + nf * per_out + (12 if kind == "best" else 0))
    if kind == "harmonics":
        nbytes += nf * 8  # the frequencies
    if kind in ("direct", "harmonics", "nfft64"):
        # one multiply-add per real sum, point and frequency
        sums = {"direct": 6, "nfft64": 2}.get(kind, 6 * case.get("nharms", 1))
        flops = c * n * nf * sums * 2
    else:
        grids = 1 if kind == "nfft" else 3
        flops = c * grids * (5.0 * nf * math.log2(max(nf, 2)) + 2 * n)
    return {"bytes": float(nbytes), "flops": float(flops)}


# ---------------------------------------------------------------------------
# the outputs in 64 bits
# ---------------------------------------------------------------------------
def _sums64(x, cid, nc, values, kc, nf):
    """sum_j v_j exp(2 pi i (kc + k') x_j), k' = -nf//2 .. nf - nf//2 - 1, of
    each of nc curves: a Gaussian-window NFFT wholly in FP64, oversampled at
    least 4 times with 28 taps (its truncation error is below 1e-15)."""
    m, G = 14, 1 << max(6, math.ceil(math.log2(4 * nf)))
    sigma = G / nf
    b = 2.0 * sigma * m / ((2.0 * sigma - 1.0) * math.pi)
    th = kc[cid] * x
    ph = torch.polar(torch.ones_like(x), 2 * math.pi * (th - torch.floor(th)))
    u = (x - torch.floor(x)) * G
    cell = torch.floor(u)
    frac = u - cell
    d = torch.arange(1 - m, m + 1, device=x.device)
    idx = (cid[:, None] * G + (cell.long()[:, None] + d[None, :]) % G).reshape(-1)
    taps = torch.exp(-(d[None, :] - frac[:, None]) ** 2 / b)
    h = nf // 2
    kp = torch.arange(-h, nf - h, device=x.device)
    dec = torch.exp(b * (math.pi * kp.double() / G) ** 2) / math.sqrt(math.pi * b)
    res = []
    for v in values:
        g = torch.zeros(nc * G, 2, dtype=torch.float64, device=x.device)
        z = torch.view_as_real(ph * v)
        for q in range(2):
            g[:, q].index_add_(0, idx, (z[:, q][:, None] * taps).reshape(-1))
        F = torch.fft.ifft(torch.view_as_complex(g).view(nc, G), dim=1, norm="forward")
        res.append(F[:, kp % G] * dec)
    return res


def _power64(YC, YS, C, S, C2, S2, mode, reg, wsum, ywsum, ybar, norm):
    """Power of the sinusoid fit from its sums (2 x 2 normal equations)."""
    if mode == "floating":
        YC, YS = YC - ywsum * C, YS - ywsum * S
        CC, SS = 0.5 * (wsum + C2) - C * C + reg, 0.5 * (wsum - C2) - S * S + reg
        CS = 0.5 * S2 - C * S
    elif mode == "standard":
        YC, YS = YC + ybar * C, YS + ybar * S
        CC, SS, CS = 0.5 * (1 + C2) + reg, 0.5 * (1 - C2) + reg, 0.5 * S2
    else:
        YC, YS = 2 * C, 2 * S
        CC, SS, CS = 0.5 * (1 + C2), 0.5 * (1 - C2), 0.5 * S2
    P = (YC * YC * SS - 2 * YC * YS * CS + YS * YS * CC) / (CC * SS - CS * CS) * norm
    return torch.where((P >= 0) & torch.isfinite(P), P, torch.full_like(P, -1.0))


def _gls64(case, b):
    """Powers of every curve, or its best power, in chunks of curves."""
    p = _prepare_host(b)
    rounded = case["kind"] in ("prepared", "direct")
    yw = p["yw"].astype(np.float64) if rounded else p["yw64"]
    w = p["w"].astype(np.float64) if rounded else p["w64"]
    ywsum = p["yw_sum"] if rounded else np.add.reduceat(yw, b["off"][:-1])
    wsum = p["w_sum"] if rounded else np.ones(len(b["N"]))
    mode, reg, out = case["mode"], _reg(case), []
    i, c = 0, case["curves"]
    while i < c:
        nf = int(b["nf"][i])
        j, room = i + 1, max(1, int(3e7 / nf))
        while j < c and j - i < room and int(b["nf"][j]) == nf:
            j += 1
        q = slice(int(b["off"][i]), int(b["off"][j]))
        cid = _dev(b["cid"][q] - i)
        x = _dev((b["t"][q] - b["t"][b["off"][:-1]][b["cid"][q]]) * b["df"][b["cid"][q]])
        kc = torch.full((j - i,), float(b["k0"] + nf // 2), dtype=torch.float64, device="cuda")
        ya, wa = _dev(yw[q]), _dev(w[q])
        A, B = _sums64(x, cid, j - i, [ya, wa], kc, nf)
        # the sums of w at twice the frequencies: the same band on 2 x
        (Cz,) = _sums64(2.0 * x, cid, j - i, [wa], kc, nf)

        def col(a):
            return _dev(np.asarray(a[i:j], np.float64))[:, None]

        norm = 1.0
        if mode == "floating":
            norm = 1.0 / col(p["yy"])
        elif mode == "standard":
            norm = 1.0 / (col(p["yy"]) + col(p["ybar"]) ** 2)
        P = _power64(A.real, A.imag, B.real, B.imag, Cz.real, Cz.imag, mode, reg, col(wsum),
                     col(ywsum), col(p["ybar"]), norm)
        out.append(P.max(dim=1).values if case["kind"] == "best" else P.reshape(-1))
        i = j
    return out


def _phases(t, f, chunk):
    """frac(t f) of every point against chunks of frequencies, the product
    kept to twice the precision (Dekker's splitting)."""
    def split(a):
        z = a * 134217729.0
        hi = z - (z - a)
        return hi, a - hi

    th, tl = split(t[:, None])
    for i in range(0, f.numel(), chunk):
        g = f[i:i + chunk][None, :]
        gh, gl = split(g)
        p = t[:, None] * g
        e = ((th * gh - p) + th * gl + tl * gh) + tl * gl
        yield (p - torch.floor(p)) + e


def _harmonics64(b, H):
    p = _prepare_host(b)
    t, yw, w = _dev(p["t"]), _dev(p["yw64"]), _dev(p["w64"])
    f = float(b["df"][0]) * (FIRST_HARMONIC_BIN
                             + torch.arange(int(b["nf"][0]), device="cuda", dtype=torch.float64))
    ybar, out = float(np.sum(p["yw64"])), []
    for ph in _phases(t, f, max(1, int(2e7 / t.numel()))):
        z = torch.polar(torch.ones_like(ph), 2 * math.pi * ph)
        W, Y, zn = [w.sum() + 0j * z[0]], [None], torch.ones_like(z)
        for n in range(1, 2 * H + 1):
            zn = zn * z
            W.append((w[:, None] * zn).sum(0))
            Y.append((yw[:, None] * zn).sum(0))
        M = torch.zeros(z.shape[1], 2 * H, 2 * H, dtype=torch.float64, device="cuda")
        r = torch.zeros(z.shape[1], 2 * H, dtype=torch.float64, device="cuda")
        for a in range(1, H + 1):
            for d in range(1, H + 1):
                lo = W[abs(a - d)]
                sg = (a > d) - (a < d)
                M[:, a - 1, d - 1] = 0.5 * (W[a + d].real + lo.real) - W[a].real * W[d].real
                cs = 0.5 * (W[a + d].imag - sg * lo.imag) - W[a].real * W[d].imag
                M[:, a - 1, H + d - 1] = cs
                M[:, H + d - 1, a - 1] = cs
                M[:, H + a - 1, H + d - 1] = (0.5 * (lo.real - W[a + d].real)
                                             - W[a].imag * W[d].imag)
            r[:, a - 1] = Y[a].real - ybar * W[a].real
            r[:, H + a - 1] = Y[a].imag - ybar * W[a].imag
        th = torch.linalg.solve(M, r)
        out.append((2 * (th * r).sum(1) - torch.einsum("ki,kij,kj->k", th, M, th)) / p["yy"][0])
    return torch.cat(out)


def exact(case, seed):
    kind = case["kind"]
    b = _batch(case, seed)
    if kind == "harmonics":
        return _harmonics64(b, case["nharms"])
    if kind in ("nfft", "nfft64"):
        out = []
        for i in range(case["curves"]):
            q = slice(int(b["off"][i]), int(b["off"][i + 1]))
            t, y = b["t"][q], b["y"][q]
            nf = int(b["nf"][i])
            if kind == "nfft64":
                # the process's grid: first frequency 0, df from the time span
                df = 1.0 / (5 * (t.max() - t.min()))
                f = df * torch.arange(nf, device="cuda", dtype=torch.float64)
                td, yd = _dev(t), _dev(y)
                out.append(torch.cat([
                    (yd[:, None] * torch.polar(torch.ones_like(ph), 2 * math.pi * ph)).sum(0)
                    for ph in _phases(td, f, max(1, int(2e7 / len(t))))]))
                continue
            df = float(b["df"][i])
            yd = _dev(y.astype(np.float32).astype(np.float64))
            x = _dev((t - t[0]) * df)
            kc = torch.full((1,), float(b["k0"] + nf // 2), dtype=torch.float64, device="cuda")
            (F,) = _sums64(x, torch.zeros(len(t), dtype=torch.long, device="cuda"), 1, [yd], kc, nf)
            th = (b["k0"] + torch.arange(nf, device="cuda", dtype=torch.float64)) * (df * t[0])
            out.append(F[0] * torch.polar(torch.ones_like(th), 2 * math.pi * (th - torch.floor(th))))
        return out if kind == "nfft64" else torch.cat(out)
    out = _gls64(case, b)
    if kind == "best":
        return (None, torch.cat(out))
    if kind == "run":
        return [q for o in out for q in o.view(-1, case["nf"])]
    return torch.cat(out)
