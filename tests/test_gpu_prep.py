"""Preparation of the curves at the edges of its length classes (one CTA up to
1,024 points, a cluster up to 8,192, a cluster of wide CTAs up to 32,768, the
chain of segment kernels above), with curves of several plans prepared in one
launch, and positions far from the usual ones (unsorted times, a first point
in the middle, x = (t - t0) df beyond a turn)."""
import numpy as np
import pytest

from test_gpu_raw import _prepared, _raw

pytestmark = pytest.mark.gpu

EDGES = [1, 2, 255, 1023, 1024, 1025, 2049, 8191, 8192, 8193, 12289, 32767, 32768, 32769, 70001]


def _curve(n, seed, T=900.0, t0=0.0):
    rng = np.random.default_rng(seed)
    t = t0 + np.sort(rng.uniform(0, T, n))
    y = 3.0 + 0.3 * np.sin(2 * np.pi * (t - t0) / 2.7) + rng.normal(0, 0.1, n)
    dy = np.exp(rng.normal(np.log(0.05), 0.3, n))
    return t, y, dy, 1.0 / (5 * T)


def _oracle_powers(oracle, c, k):
    t, y, dy, df = c
    tt, yw, w, YY, _ = oracle.prepare_curve(t, y, dy)
    return oracle.gls_flmean(tt, yw, w, df * (1 + k), YY)


@pytest.fixture(scope="module", params=["mixed", "fp32", "auto"])
def h(request):
    from cuvarbase_gb300 import _lib
    hh = _lib.Handle(sigma=-1.0 if request.param == "auto" else 2.0, m=8,
                     precision=_lib.PREC_FP32 if request.param == "fp32" else _lib.PREC_MIXED)
    hh.tol = {"mixed": 1e-5, "fp32": 5e-3, "auto": 1e-4}[request.param]
    yield hh
    hh.close()


@pytest.mark.parametrize("raw", [True, False])
def test_length_classes_in_one_call(h, oracle, raw):
    curves = [_curve(n, 100 + n) for n in EDGES]
    nf = 3000
    P = (_raw if raw else _prepared)(h, curves, nf)
    for c, got in zip(curves, P):
        if len(c[0]) < 200:
            continue          # nearly exact fits: the denominator is rounding
        k = np.arange(50, nf, 7)
        assert np.abs(got[k] - _oracle_powers(oracle, c, k)).max() <= h.tol


def test_several_plans_in_one_call(oracle):
    """Curves of many frequency counts (and so plans) in one call: the same
    as each alone, with host and with device buffers."""
    from cuvarbase_gb300.lombscargle import LombScargleAsyncProcess
    sizes = [(300, 700), (1500, 40000), (9000, 3000), (40, 90000), (40000, 5000), (2000, 250000),
             (1024, 12000), (700, 700)]
    data = [_curve(n, 7 + n)[:3] for n, _ in sizes]
    freqs = [(1 + np.arange(nf)) / (5 * 900.0) for _, nf in sizes]
    for sigma in ("auto", 2):
        p = LombScargleAsyncProcess(sigma=sigma, m=8)
        got = p.run(data, freqs=freqs)
        p.finish()
        got = [np.copy(P) for _, P in got]
        for d, f, P in zip(data, freqs, got):
            (_, alone), = p.run([d], freqs=[f])
            p.finish()
            tt, yw, w, YY, _ = oracle.prepare_curve(*d)
            k = np.arange(20, len(f), max(1, len(f) // 300))
            ref = oracle.gls_flmean(tt, yw, w, f[k], YY)
            assert np.abs(P[k] - ref).max() <= 1e-4
            # the order of the atomic adds differs from run to run
            assert np.abs(P - alone).max() <= 2e-5


@pytest.mark.parametrize("raw", [True, False])
def test_short_curves_of_a_large_batch(oracle, raw):
    """The class of short curves, which only a batch that fills the chip uses:
    the edges of its sizes, beside longer curves."""
    from cuvarbase_gb300 import _lib
    from test_gpu_rows import _ref
    sizes = ([1, 2, 63, 64, 65, 127, 383, 384, 385, 1024, 3000] * 70)
    curves = [_curve(n, 31 * i + n) for i, n in enumerate(sizes)]
    hh = _lib.Handle(sigma=2.0, m=8)
    try:
        nf = 500
        k = np.arange(50, nf, 3)
        for mode in (2, 1) if raw else (1,):
            P = _raw(hh, curves, nf, mode) if raw else _prepared(hh, curves, nf)
            for i in list(range(11)) + [400, 401, 402, 403, 404, 767, 768, 769]:
                n = len(curves[i][0])
                if n < 3 or (mode == 1 and n < 200):
                    continue      # singular; nearly exact fits: rounding over rounding
                ref = _ref(oracle, curves[i], k, mode)
                assert np.abs(P[i][k] - ref).max() <= 2e-5 * max(1.0, np.abs(ref).max())
    finally:
        hh.close()


@pytest.mark.parametrize("n", [300, 1500, 20000, 40000])
def test_unsorted_and_far_times(oracle, n):
    """Positions of every sign and many turns: shuffled times, an origin far
    away, and a grid whose df T is 37 turns."""
    from cuvarbase_gb300 import _lib
    rng = np.random.default_rng(n)
    t, y, dy, _ = _curve(n, n, t0=-4.0e5)
    q = rng.permutation(n)
    df = 37.0 / 900.0
    c = (t[q], y[q], dy[q], df)
    hh = _lib.Handle(sigma=2.0, m=8)
    try:
        for f in (_raw, _prepared):
            P = f(hh, [c], 2000)[0]
            k = np.arange(0, 2000, 3)
            assert np.abs(P[k] - _oracle_powers(oracle, c, k)).max() <= 2e-5
    finally:
        hh.close()


@pytest.mark.parametrize("n", [100, 1500, 20000, 40000])
def test_first_time_not_finite(n):
    """A first time that is not finite leaves no valid power in its curve and
    the other curves alone."""
    from cuvarbase_gb300 import _lib
    good = _curve(500, 1)
    t, y, dy, df = _curve(n, 2)
    t = t.copy()
    t[0] = np.nan
    hh = _lib.Handle(sigma=2.0, m=8)
    try:
        P = _raw(hh, [good, (t, y, dy, df)], 2000)
        assert np.all(P[1] == -1.0)
        assert np.abs(P[0] - _raw(hh, [good], 2000)[0]).max() <= 1e-6
        assert hh.device_flags() & _lib.DEVERR_NONFINITE
    finally:
        hh.close()


@pytest.mark.parametrize("f0", [0.0, 1.2345])
def test_nfft_length_classes(oracle, f0):
    """f0 / df is not a whole number in the second case."""
    from cuvarbase_gb300.cunfft import NFFTAsyncProcess
    data = [(t - 300.0, y, 2500) for t, y, _, _ in (_curve(n, n) for n in EDGES[2:])]
    p = NFFTAsyncProcess(sigma=2, m=8)
    res = p.run(data, minimum_frequency=f0, samples_per_peak=3)
    p.finish()
    for (t, y, nf), got in zip(data, res):
        df = 1.0 / (3 * (t.max() - t.min()))
        k = np.arange(0, nf, 9)
        ref = oracle.nfft_direct(t, y, f0 + k * df)
        assert np.abs(got[k] - ref).max() <= 2e-6 * np.abs(y).sum()
