"""Tiles that threads write and a bulk copy then refills.  The copies belong to
the async proxy, and a barrier orders only the threads' own accesses, so every
barrier before such a refill is preceded by the proxy fence.  (Nothing a GPU
computes shows a missing one; the first test reads the source.)"""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuvarbase_gb300",
                    "csrc")


def test_proxy_fence_before_every_refill():
    src = open(os.path.join(CSRC, "pass2_tma.cuh")).read()
    src = re.sub(r"//[^\n]*", "", src)
    helper = re.search(r"void (\w+)\(\) \{\s*asm volatile\(\"fence\.proxy\.async\.shared::cta;\"", src)
    assert helper
    refills = re.findall(r"([^;{}]*;)\s*__syncthreads\(\);\s*if \(tid == 0\) issue\(", src)
    assert len(refills) == 2          # the two kernels that exchange in place
    for before in refills:
        assert before.strip() == helper.group(1) + "();"


@pytest.mark.gpu
@pytest.mark.parametrize("sigma", [2.0, 4.0])
@pytest.mark.parametrize("G2", [160, 256, 320, 400])
def test_gls_many_tiles_per_cta(G2, sigma):
    """The same curve many times over, so that every persistent CTA refills
    its tile several times: one set of powers."""
    from cuvarbase_gb300 import _lib
    from test_gpu_prep import _curve
    from test_gpu_raw import _raw
    G1, n = 160, 250                  # 2,500 to 5,000 tiles for at most 608 CTAs
    h = _lib.Handle(sigma=sigma, m=8)
    try:
        nf = int(G1 * G2 / sigma)
        h.plan_pin(nf, G1, G2)
        P = _raw(h, [_curve(300, G2)] * n, nf)
        # the order of the atomic adds differs from curve to curve
        assert max(np.abs(p - P[0]).max() for p in P) <= 2e-5
    finally:
        h.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nf", [2500, 5000, 12800, 31000, 50000, 100000])
def test_nfft_many_tiles_per_cta(nf):
    from cuvarbase_gb300.cunfft import NFFTAsyncProcess
    from test_gpu_prep import _curve
    t, y, _, _ = _curve(300, nf)
    p = NFFTAsyncProcess(sigma=2, m=8)
    res = p.run([(t, y, nf)] * 300, samples_per_peak=3)
    p.finish()
    assert max(np.abs(r - res[0]).max() for r in res) <= 2e-6 * np.abs(y).sum()
