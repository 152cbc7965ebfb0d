"""The 64-bit direct-sum kernels at the edges of their tiles: bins per CTA (416
for the NFFT, 224 for the GLS, 32 frequencies for the harmonics), points per
warp and per CTA (32, 256), one part and several parts of the points, against
the FP64 oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


def curve(n, seed):
    rng = np.random.default_rng(seed)
    t = np.sort(rng.uniform(0, 1000, n))
    t[0] = 0.0
    y = np.sin(2 * np.pi * t / 3.3 + 0.4) + 0.1 * rng.standard_normal(n)
    return t, y, np.exp(rng.normal(np.log(0.05), 0.3, n))


@pytest.mark.parametrize("sizes", [
    [(2, 1), (3, 543), (31, 544)], [(32, 545), (33, 17)], [(256, 1088), (257, 1089)],
    [(1025, 3000), (255, 2999)],
    [(40, 415), (41, 416)], [(70, 417), (300, 833)],
    [(40 + i, 20000) for i in range(40)],        # enough CTAs: one part
    [(70, 700000)],
])
def test_use_double_tiles(oracle, sizes):
    from cuvarbase_gb300.cunfft import NFFTAsyncProcess
    data = [curve(n, 10 + i)[:2] + (nf,) for i, (n, nf) in enumerate(sizes)]
    p = NFFTAsyncProcess(use_double=True)
    res = p.run(data, samples_per_peak=5, minimum_frequency=0.3)
    p.finish()
    for (t, y, nf), got in zip(data, res):
        df = 1.0 / (5 * (t.max() - t.min()))
        f = 0.3 + df * np.arange(nf)
        ref = oracle.nfft_direct(t, y, f)
        # phase rounding of both sides (a few units of f t), then the sums
        tol = np.abs(y).sum() * EPS * (8 * 2 * np.pi * (1 + f[-1] * t.max()) + len(t))
        assert np.abs(got - ref).max() <= tol


@pytest.mark.parametrize("scale", [1e300, 1e-300, 5e-324 * 2 ** 20, 0.0, "mixed"])
def test_use_double_scales(oracle, scale):
    """Values near the ends of the double range, all zero, and over 24 orders
    of magnitude in one curve."""
    from cuvarbase_gb300.cunfft import NFFTAsyncProcess
    t, y, _ = curve(300, 8)
    y = y * 10.0 ** np.random.default_rng(9).uniform(-12, 12, 300) if scale == "mixed" else y * scale
    p = NFFTAsyncProcess(use_double=True)
    (got,) = p.run([(t, y, 500)], samples_per_peak=5, minimum_frequency=0.3)
    p.finish()
    f = 0.3 + np.arange(500) / (5 * (t.max() - t.min()))
    # the oracle on values of order one (times the exact power of two; a value
    # below the normal range is a whole number of the smallest one)
    ex = 0 if scale in (0.0, "mixed") else int(np.floor(np.log2(np.abs(y).max())))
    ref = oracle.nfft_direct(t, np.ldexp(y, -ex), f)
    got = np.ldexp(got.real, -ex) + 1j * np.ldexp(got.imag, -ex)
    tol = np.abs(np.ldexp(y, -ex)).sum() * EPS * (8 * 2 * np.pi * (1 + f[-1] * t.max()) + 300)
    if ex < -1000:
        # each of the two parts' real and imaginary sums rounds to half a unit
        tol += 2 * np.sqrt(0.5) * np.ldexp(1.0, -1074 - ex)
    assert np.abs(got - ref).max() <= tol


def test_long_parts(oracle):
    """More points per warp than one run of integer sums holds (enough bins
    that the points are not cut into parts)."""
    from cuvarbase_gb300.cunfft import NFFTAsyncProcess
    from cuvarbase_gb300.lombscargle import LombScargleAsyncProcess
    n, nf = 17000, 520000
    t, y, dy = curve(n, 4)
    k = np.unique(np.concatenate([np.arange(20, 60), np.arange(nf - 40, nf), np.arange(21, nf, 9001)]))
    p = NFFTAsyncProcess(use_double=True)
    (got,) = p.run([(t, y, nf)], samples_per_peak=5, minimum_frequency=0.3)
    p.finish()
    f = 0.3 + k / (5 * (t.max() - t.min()))
    ref = oracle.nfft_direct(t, y, f)
    tol = np.abs(y).sum() * EPS * (8 * 2 * np.pi * (1 + f[-1] * t.max()) + n)
    assert np.abs(got[k] - ref).max() <= tol
    p = LombScargleAsyncProcess(sigma=2, m=8)
    f = (1 + np.arange(nf)) / (5 * (t.max() - t.min()))
    ((_, got),) = p.run([(t, y, dy)], freqs=[f], use_fft=False)
    p.finish()
    tt, yw, w, YY, ybar = oracle.prepare_curve(t, y, dy)
    ref = oracle.gls_tau(tt, yw.astype(np.float32).astype(np.float64),
                         w.astype(np.float32).astype(np.float64), f[k], YY, ybar, mode=1)
    assert np.abs(got[k] - ref).max() <= 2e-6 * max(1.0, np.abs(ref).max())


def test_use_double_infinite_value():
    """An infinite value makes every bin infinite with the signs of its own
    phase, not NaN."""
    from cuvarbase_gb300.cunfft import NFFTAsyncProcess
    t, y, _ = curve(100, 3)
    y[40] = np.inf
    p = NFFTAsyncProcess(use_double=True)
    (got,) = p.run([(t, y, 50)], samples_per_peak=5)
    p.finish()
    th = 2 * np.pi * t[40] * np.arange(1, 50) / (5 * (t.max() - t.min()))
    assert np.array_equal(got.real[1:], np.copysign(np.inf, np.cos(th)))
    assert np.array_equal(got.imag[1:], np.copysign(np.inf, np.sin(th)))


@pytest.mark.parametrize("mode", ["floating", "standard", "window"])
@pytest.mark.parametrize("sizes", [
    [(20, 2), (31, 287), (32, 288)], [(33, 289), (256, 577)], [(1025, 2000), (300, 1999)],
    [(30 + i, 10000) for i in range(40)],        # enough CTAs: one part
])
def test_direct_sums_tiles(oracle, sizes, mode):
    from cuvarbase_gb300.lombscargle import LombScargleAsyncProcess
    data = [curve(n, 30 + i) for i, (n, _) in enumerate(sizes)]
    freqs = [(20 + np.arange(nf)) / (5 * (t.max() - t.min()))
             for (t, _, _), (_, nf) in zip(data, sizes)]
    p = LombScargleAsyncProcess(sigma=2, m=8)
    kw = dict(floating_mean=mode != "standard", window=mode == "window")
    res = p.run(data, freqs=freqs, use_fft=False, **kw)
    p.finish()
    num = {"standard": 0, "floating": 1, "window": 2}[mode]
    for (t, y, dy), f, (_, got) in zip(data, freqs, res):
        tt, yw, w, YY, ybar = oracle.prepare_curve(t, y, dy)
        ref = oracle.gls_tau(tt, yw.astype(np.float32).astype(np.float64),
                             w.astype(np.float32).astype(np.float64), f, YY, ybar, mode=num)
        # float32 results, yw and w the same float32 values on both sides; the
        # statistics of the curve are float32 in the kernel
        assert np.abs(got - ref).max() <= 2e-6 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("H", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("n,nf", [(40, 1), (255, 31), (256, 32), (257, 33), (1000, 100)])
def test_harmonics_tiles(oracle, H, n, nf):
    from cuvarbase_gb300.lombscargle import lomb_scargle_direct_sums
    t, y, dy = curve(n, 5 * H)
    tt, yw, w, YY, _ = oracle.prepare_curve(t, y, dy)
    f = (12 + np.arange(nf)) / (5 * (t.max() - t.min()))
    f[-1] = 1 / 3.3
    P = lomb_scargle_direct_sums(tt, yw, w, f, YY, nharms=H, amplitude_priors=3.0)
    ref = oracle.mhgls_np(tt, yw, w, f, YY, nharms=H, amplitude_priors=3.0)
    assert np.abs(P - ref).max() <= 1e-9


def test_harmonics_large_phases(oracle):
    """Phases beyond 2^40 turns (times given with a far origin) still follow
    frac(t f) of the FP64 product."""
    from cuvarbase_gb300.lombscargle import lomb_scargle_direct_sums
    t, y, dy = curve(200, 77)
    _, yw, w, YY, _ = oracle.prepare_curve(t, y, dy)
    t = t + 2.0 ** 38
    f = np.array([16.5, 17.25])
    P = lomb_scargle_direct_sums(t, yw, w, f, YY, nharms=2, amplitude_priors=3.0)
    ref = oracle.mhgls_np(t, yw, w, f, YY, nharms=2, amplitude_priors=3.0)
    assert np.abs(P - ref).max() <= 1e-9


@pytest.mark.parametrize("H", [1, 3])
def test_harmonics_long_curve(oracle, H):
    """More points per warp than one run of integer sums holds, and weights
    over six orders of magnitude."""
    from cuvarbase_gb300.lombscargle import lomb_scargle_direct_sums
    t, y, dy = curve(40000, 6)
    dy = dy * 10.0 ** np.random.default_rng(5).uniform(0, 3, len(t))
    tt, yw, w, YY, _ = oracle.prepare_curve(t, y, dy)
    f = (12 + np.arange(40)) / (5 * (t.max() - t.min()))
    f[-1] = 1 / 3.3
    P = lomb_scargle_direct_sums(tt, yw, w, f, YY, nharms=H, amplitude_priors=3.0)
    ref = oracle.mhgls_np(tt, yw, w, f, YY, nharms=H, amplitude_priors=3.0)
    assert np.abs(P - ref).max() <= 1e-9


def test_harmonics_values_not_finite():
    """A time or weight that is not finite leaves no frequency a power, a
    frequency that is not finite none of its own."""
    from cuvarbase_gb300.lombscargle import lomb_scargle_direct_sums
    t, y, _ = curve(600, 2)
    w = np.full(600, 1 / 600)
    f = np.linspace(0.1, 2.0, 70)

    def put(a, i, v):
        a = a.copy()
        a[i] = v
        return a
    for v in (np.nan, np.inf):
        for args in ((put(t, 7, v), w * y, w, f), (t, w * y, put(w, 7, v), f)):
            assert np.all(np.isnan(lomb_scargle_direct_sums(*args, 1.0, nharms=2)))
        P = lomb_scargle_direct_sums(t, w * y, w, put(f, 5, v), 1.0, nharms=2)
        assert np.isnan(P[5]) and np.isfinite(np.delete(P, 5)).all()
