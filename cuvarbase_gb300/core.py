"""Asynchronous-process base class (mirrors cuvarbase/core.py:13-56)."""
from __future__ import annotations

from . import _lib


class ResultPool:
    """Page-locked buffers for the results of one process.  Page-locking a
    megabyte takes a few hundred microseconds, longer than most calls' kernels,
    so buffers whose results are gone are kept, the last ``KEEP`` of them; the
    others are given back at once.  A result takes no buffer of more than twice
    its size (or a megabyte), so that results which a program keeps hold little
    more than themselves."""

    KEEP = 4
    SMALL = 1 << 20

    def __init__(self):
        self._free = []

    def take(self, nbytes):
        """A lease on a buffer of at least nbytes."""
        nbytes = (max(int(nbytes), 1) + 4095) // 4096 * 4096
        fit = [b for b in list(self._free)
               if nbytes <= b.nbytes <= max(2 * nbytes, self.SMALL)]
        for buf in sorted(fit, key=lambda b: b.nbytes):
            try:
                self._free.remove(buf)
            except ValueError:  # taken by another thread
                continue
            break
        else:
            buf = _lib.PinnedBuffer(nbytes)
        return ResultBuffer(self, buf)

    def give(self, buf):
        self._free.append(buf)
        del self._free[:-self.KEEP]


class ResultBuffer:
    """A lease on a page-locked buffer; it ends with the last view."""

    def __init__(self, pool, buf):
        self._pool, self._buf = pool, buf
        self.ptr, self.nbytes = buf.ptr, buf.nbytes

    def view(self, dtype, count, offset_bytes=0):
        return self._buf.view(dtype, count, offset_bytes, owner=self)

    def __del__(self):
        self._pool.give(self._buf)


class GPUAsyncProcess:
    """Base of the GPU processes: owns CUDA streams and library handles.

    Keyword arguments as in the reference: ``nstreams``, ``device``,
    ``reader`` and ``function_kwargs``.  Unlike the reference, ``device``
    selects the GPU the handles run on.
    """

    def __init__(self, *args, **kwargs):
        self.reader = kwargs.get('reader', None)
        self.nstreams = kwargs.get('nstreams', None)
        self.function_kwargs = kwargs.get('function_kwargs', {})
        self.device = kwargs.get('device', 0)
        self.streams = []
        self.gpu_data = []
        self.results = []
        self._adjust_nstreams = self.nstreams is None
        self._handles = {}
        self._result_pool = ResultPool()
        if self.nstreams is not None:
            self._create_streams(self.nstreams)
        self.prepared_functions = {}

    def _create_streams(self, n):
        for _ in range(n):
            self.streams.append(_lib.Stream())

    def _stream(self):
        if not self.streams:
            self._create_streams(1)
        return self.streams[0]

    def _handle(self, sigma, m, precision=_lib.PREC_MIXED, workspace_bytes=0):
        key = (float(sigma), int(m), int(precision))
        h = self._handles.get(key)
        if h is None:
            h = _lib.Handle(sigma=sigma, m=m, device=self.device,
                            workspace_bytes=workspace_bytes, precision=precision)
            self._handles[key] = h
        return h

    def _result_buffer(self, nbytes):
        """A page-locked result buffer, the process's again when the last
        array that views it is gone."""
        return self._result_pool.take(nbytes)

    def _compile_and_prepare_functions(self, **kwargs):
        """Kernels are compiled ahead of time into libcuvgls.so; this only
        loads the library (kept for API compatibility)."""
        _lib.load()

    def run(self, *args, **kwargs):
        raise NotImplementedError()

    def finish(self, timeout_ms=-1):
        """Synchronise every stream this process used (cuvarbase/core.py:37-40).

        With ``timeout_ms >= 0`` a stuck stream raises TimeoutError instead
        of blocking forever.
        """
        for h in self._handles.values():
            for s in (self.streams or [None]):
                h.sync(None if s is None else s.ptr, timeout_ms)

    def batched_run(self, data, batch_size=10, **kwargs):
        """run() on consecutive batches of ``batch_size`` light curves, with a
        finish() after each (cuvarbase/core.py:42-56)."""
        nsubmit = 0
        results = []
        while nsubmit < len(data):
            batch = []
            while len(batch) < batch_size and nsubmit < len(data):
                batch.append(data[nsubmit])
                nsubmit += 1
            res = self.run(batch, **kwargs)
            self.finish()
            results.extend(res)
        return results
