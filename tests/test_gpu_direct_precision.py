"""The 64-bit direct sums with one value that dominates a long curve: no coarser
than the same sums in FP64.  Times, frequencies and their products are exact, so
that the sums are all that rounds."""
import numpy as np
import pytest

LD = np.longdouble
TWO_PI = 2 * LD("3.14159265358979323846264338327950288")


def _curve(n, seed):
    """Times of 30 bits over 1,024; a value of nearly 2 among ones of 10^-3."""
    rng = np.random.default_rng(seed)
    t = np.sort(rng.integers(1, (1 << 30) - 1, n)) / 2.0 ** 20
    t[0], t[-1] = 0.0, 1024.0
    y = rng.standard_normal(n) * 1e-3
    y[n // 7] = 1.98
    return t, y


def _sums(t, v, f):
    """sum v exp(2 pi i t f) per frequency, in extended precision."""
    out = np.empty((len(f), 2), LD)
    for i, x in enumerate(f):
        ph = t * x                       # exact
        a = TWO_PI * (ph - np.floor(ph)).astype(LD)
        out[i] = (v.astype(LD) * np.cos(a)).sum(), (v.astype(LD) * np.sin(a)).sum()
    return out


def _rms_fp64(n):
    """A sum in FP64 that holds a value in [1, 2) rounds to units of 2^-52: 0.29
    of them per addition (rms)."""
    return 0.29 * 2.0 ** -52 * np.sqrt(n)


@pytest.mark.gpu
@pytest.mark.parametrize("n,nf", [(300, 400), (2000, 520000), (8192, 520000)])
def test_use_double_one_value_dominates(n, nf):
    """Both with the points in parts and, with enough bins, in one part."""
    from cuvarbase_gb300.cunfft import NFFTAsyncProcess
    t, y = _curve(n, n)
    p = NFFTAsyncProcess(use_double=True)
    (got,) = p.run([(t, y, nf)], samples_per_peak=1)
    p.finish()
    k = np.random.default_rng(1).integers(0, nf, 120)
    ref = _sums(t, y, k / 1024.0)
    err = np.concatenate([got.real[k] - ref[:, 0], got.imag[k] - ref[:, 1]]).astype(float)
    assert np.sqrt(np.mean(err ** 2)) <= _rms_fp64(n)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [500, 2000, 32768])
def test_harmonics_one_value_dominates(n):
    from cuvarbase_gb300.lombscargle import lomb_scargle_direct_sums
    t, yw = _curve(n, n + 1)
    w = np.full(n, 2.0 ** -20)           # exact, as is their sum
    f = np.random.default_rng(2).integers(1 << 12, 1 << 18, 96) / 1024.0
    P = lomb_scargle_direct_sums(t, yw, w, f, 1.0, nharms=1)
    W = n * LD(2) ** -20
    C, S = _sums(t, w, f).T
    C2, S2 = _sums(t, w, 2 * f).T
    YC, YS = (_sums(t, yw, f) - LD(np.cumsum(yw)[-1]) * _sums(t, w, f)).T
    CC, SS, CS = (W + C2) / 2 - C * C, (W - C2) / 2 - S * S, S2 / 2 - C * S
    ref = (YC * YC * SS - 2 * YC * YS * CS + YS * YS * CC) / (CC * SS - CS * CS)
    # P goes as the squares of YC and YS, whose larger one is 1.4 or more
    err = ((P - ref) / ref).astype(float)
    assert np.sqrt(np.mean(err ** 2)) <= 2 * _rms_fp64(n) / 1.4 + 16 * 2.0 ** -53


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [np.nan, np.inf, 1e30])
def test_window_needs_no_values(bad):
    """The spectral window (mode "window") is that of the weights: a value that
    is not finite, or not in float32, leaves its powers alone; in the other
    modes it leaves the curve none."""
    import ctypes
    from cuvarbase_gb300 import _lib
    rng = np.random.default_rng(7)
    n, nf = 300, 700
    t = np.sort(rng.uniform(0, 900.0, n))
    w = np.full(n, 1 / n, np.float32)
    yw = (rng.standard_normal(n) / n).astype(np.float32)

    def powers(yw, mode):
        c = _lib.Curve()
        c.pt_off, c.n, c.nf, c.k0, c.df, c.out_off = 0, n, nf, 1, 1 / 4500.0, 0
        c.yy, c.ybar, c.yw_sum, c.w_sum = 1.0, 0.0, float(yw.sum()), float(w.sum())
        inp = _lib.GlsInput()
        inp.n_curves, inp.mode = 1, mode
        inp.curves = ctypes.addressof(c)
        inp.t, inp.yw, inp.w = t.ctypes.data, yw.ctypes.data, w.ctypes.data
        inp.flags = _lib.HOST_INPUT | _lib.HOST_OUTPUT
        inp.n_points_total, inp.n_out_total = n, nf
        P = np.empty(nf, np.float32)
        h.check(_lib.load().cuvgls_gls_direct_batch(h.ptr, ctypes.byref(inp), P.ctypes.data, None),
                "direct")
        h.sync(None, -1)
        return P
    h = _lib.Handle(sigma=2.0, m=8)
    try:
        spoilt = yw.copy()
        with np.errstate(over="ignore"):
            spoilt[11] = np.float32(bad) * np.float32(1e10)
        want = powers(yw, _lib.MODE_WINDOW)
        assert np.all(want >= 0)
        assert np.array_equal(powers(spoilt, _lib.MODE_WINDOW), want)
        for mode in (_lib.MODE_STANDARD, _lib.MODE_FLOATING_MEAN):
            assert np.all(powers(spoilt, mode) == -1)
    finally:
        h.close()
