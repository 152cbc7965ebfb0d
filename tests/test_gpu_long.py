"""Pass 1 of the GLS at the long column lengths: column blocks with no record,
a few, and more than one round of them per thread, records around the wrap of
rows and columns, narrow and wide grids, both windows, against the FP64
oracle."""
import numpy as np
import pytest

from test_gpu_prep import _curve
from test_gpu_raw import _raw
from test_gpu_rows import _ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G2", [32, 80, 400])
@pytest.mark.parametrize("G1", [1280, 1600, 2048])
def test_long_columns(oracle, G1, G2):
    from cuvarbase_gb300 import _lib
    curves = [_curve(n, n + G1) for n in (5, 300, 40000)]
    # the tolerances of the other lengths: ES budget, FP32 rounding of the Gaussian
    for sigma, tol in ((-1.0, 1e-4), (2.0, 2e-5)):
        h = _lib.Handle(sigma=sigma, m=8)
        try:
            nf = int(G1 * G2 / (1.28 if sigma < 0 else 2.0))
            h.plan_pin(nf, G1, G2)
            assert h.plan(nf)[1:3] == (G1, G2)
            k = np.unique(np.concatenate([np.arange(30, 90), np.arange(nf - 60, nf),
                                          np.arange(31, nf, max(1, nf // 60))]))
            for mode in (2, 1):
                P = _raw(h, curves, nf, mode)
                for c, got in zip(curves, P):
                    # (five points and three parameters: the normal equations
                    # come close to singular, the spectral window does not)
                    if mode == 1 and len(c[0]) == 5:
                        continue
                    ref = _ref(oracle, c, k, mode)
                    assert np.abs(got[k] - ref).max() <= tol * max(1.0, np.abs(ref).max())
        finally:
            h.close()


@pytest.mark.parametrize("G1", [16, 32, 64, 80, 128, 160, 256, 320, 400, 512, 640, 800, 1024])
def test_many_records(oracle, G1):
    """Column blocks spread record by record, beside blocks of the same launch
    that are not, at the other column lengths."""
    from cuvarbase_gb300 import _lib
    curves = [_curve(n, n + G1) for n in (9000, 300)]
    for sigma, tol in ((-1.0, 1e-4), (2.0, 2e-5)):
        h = _lib.Handle(sigma=sigma, m=8)
        try:
            G2 = 32
            nf = int(G1 * G2 / (1.28 if sigma < 0 else 2.0))
            h.plan_pin(nf, G1, G2)
            assert h.plan(nf)[1:3] == (G1, G2)
            k = np.unique(np.concatenate([np.arange(30, min(nf, 90)), np.arange(nf - 60, nf),
                                          np.arange(31, nf, max(1, nf // 60))]))
            for mode in (1, 2):
                P = _raw(h, curves, nf, mode)
                for c, got in zip(curves, P):
                    ref = _ref(oracle, c, k, mode)
                    assert np.abs(got[k] - ref).max() <= tol * max(1.0, np.abs(ref).max())
        finally:
            h.close()


@pytest.mark.parametrize("nf", [150, 400, 1000, 2500, 5000, 12800, 30000])
def test_nfft_many_records(oracle, nf):
    from cuvarbase_gb300.cunfft import NFFTAsyncProcess
    data = [(t, y, nf) for t, y, _, _ in (_curve(n, nf + n) for n in (20000, 200))]
    p = NFFTAsyncProcess(sigma=2, m=8)
    res = p.run(data, minimum_frequency=0.7531, samples_per_peak=3)
    p.finish()
    for (t, y, _), got in zip(data, res):
        df = 1.0 / (3 * (t.max() - t.min()))
        k = np.unique(np.concatenate([np.arange(40), np.arange(nf - 40, nf),
                                      np.arange(0, nf, max(1, nf // 60))]))
        ref = oracle.nfft_direct(t, y, 0.7531 + k * df)
        # FP32 rounding of the Gaussian window at the band edge, as for few points
        assert np.abs(got[k] - ref).max() <= 2e-6 * np.abs(y).sum()
