"""Page-locked result buffers of the processes: a result owns its buffer until
its last view is gone, what a program keeps holds little more than itself, and
what it drops is used again or given back."""
import ctypes
import sys
import weakref

import numpy as np
import pytest

from cuvarbase_gb300 import _lib
from cuvarbase_gb300.core import GPUAsyncProcess


class _HostBuffer(_lib.PinnedBuffer):
    """Pageable stand-in for the page-locked allocation."""
    live = weakref.WeakSet()
    made = 0

    def __init__(self, nbytes):
        self.nbytes = max(int(nbytes), 16)
        self._mem = ctypes.create_string_buffer(self.nbytes)
        self.ptr = ctypes.c_void_p(ctypes.addressof(self._mem))
        self._np = np
        _HostBuffer.live.add(self)
        _HostBuffer.made += 1

    def close(self):
        self.ptr = None


@pytest.fixture
def proc(monkeypatch):
    monkeypatch.setattr(_lib, "PinnedBuffer", _HostBuffer)
    _HostBuffer.live = weakref.WeakSet()
    _HostBuffer.made = 0
    return GPUAsyncProcess()


def _result(proc, n):
    return proc._result_buffer(8 * n).view(np.complex64, n)


def _held():
    return sum(b.nbytes for b in _HostBuffer.live)


def test_kept_results_hold_their_own_size(proc):
    kept = [_result(proc, 1000) for _ in range(200)]
    assert len(kept) * 8000 <= _held() <= len(kept) * (8000 + 4096)


def test_small_result_leaves_a_large_buffer_alone(proc):
    big = _result(proc, 8 << 20)
    del big
    small = _result(proc, 1000)
    assert small.base._owner.nbytes <= 1 << 20


def test_dropped_buffer_is_used_again(proc):
    r = _result(proc, 100000)
    part = r[5:10]
    del r
    s = _result(proc, 100000)            # the first one is still viewed
    assert _HostBuffer.made == 2
    del part, s
    for n in (100000, 99999, 60000):
        x = _result(proc, n)
        del x
    assert _HostBuffer.made == 2


@pytest.mark.parametrize("borrowed", [0, 1])
def test_held_results_are_not_written_again(proc, monkeypatch, borrowed):
    """Whatever the interpreter counts as references (some pass locals without
    one of their own)."""
    count = sys.getrefcount
    monkeypatch.setattr(sys, "getrefcount", lambda o: count(o) - 1 - borrowed)
    sizes = [3000, 3000, 2900, 500, 200000, 3000]
    kept = []
    for i, n in enumerate(sizes):
        x = _result(proc, n)
        x[:] = i
        kept.append(x)
    for i, x in enumerate(kept):
        assert np.all(x == i)


def test_free_buffers_are_bounded(proc):
    kept = [_result(proc, 50000 + i) for i in range(60)]
    assert _held() >= 60 * 400000
    del kept
    assert len(_HostBuffer.live) <= 4


@pytest.mark.gpu
def test_results_survive_later_calls():
    from cuvarbase_gb300.cunfft import NFFTAsyncProcess
    from cuvarbase_gb300.lombscargle import LombScargleAsyncProcess
    rng = np.random.default_rng(0)

    def curve(n):
        t = np.sort(rng.uniform(0, 400, n))
        return t, np.sin(t), np.full(n, 0.1)

    gls, nfft, exact = (LombScargleAsyncProcess(sigma=2, m=8), NFFTAsyncProcess(sigma=2, m=8),
                        NFFTAsyncProcess(use_double=True))
    kept = []
    for nf in (3000, 3000, 500, 150000, 3000, 2900):
        t, y, dy = curve(300)
        ((_, P),) = gls.run([(t, y, dy)], freqs=[(1 + np.arange(nf)) / 2000.0])
        gls.finish()
        kept.append((P, P.copy()))
        for p in (nfft, exact):
            (g,) = p.run([(t, y, nf)], samples_per_peak=3)
            p.finish()
            kept.append((g, g.copy()))
    for now, then in kept:
        assert np.array_equal(now, then)
