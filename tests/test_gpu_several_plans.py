"""Batches of several plans (frequency counts), whose passes run beside each
other on side streams: device buffers, captured plans, a caller's own capture,
calls on two streams in turn, and every form that a smaller workspace leads to."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# the order of the atomic adds differs from run to run
TOL = 2e-5
SIZES = [(300, 700), (1500, 40000), (9000, 3000), (40, 90000), (40000, 5000), (2000, 120000),
         (1024, 12000), (700, 700), (120, 20000)]


class Batch:
    """Curves of (points, frequencies) on the device, raw or prepared."""

    def __init__(self, sizes, seed, prepared=False):
        import torch
        from cuvarbase_gb300 import _lib
        self.sizes, self.prepared = sizes, prepared
        n, nf = (np.array([s[k] for s in sizes]) for k in (0, 1))
        self.off = np.concatenate([[0], np.cumsum(n)])
        self.out_off = np.concatenate([[0], np.cumsum(nf)])
        self.cv = ((_lib.Curve if prepared else _lib.RawCurve) * len(sizes))()
        for i, c in enumerate(self.cv):
            c.pt_off, c.n, c.nf, c.k0, c.df = int(self.off[i]), int(n[i]), int(nf[i]), 1, 1 / 4500.0
            c.out_off = int(self.out_off[i])
        self.bufs = [torch.empty(int(self.off[-1]), device="cuda",
                                 dtype=torch.float32 if prepared and k else torch.float64)
                     for k in range(3)]
        self.fill(seed)
        self.out = torch.empty(int(self.out_off[-1]), device="cuda")
        self.best = (torch.empty(len(sizes), dtype=torch.int64, device="cuda"),
                     torch.empty(len(sizes), device="cuda"))
        self.inp = (_lib.GlsInput if prepared else _lib.RawInput)()
        self.inp.n_curves, self.inp.mode, self.inp.flags = len(sizes), 1, 0
        self.inp.curves = ctypes.cast(self.cv, ctypes.c_void_p)
        ptr = [b.data_ptr() for b in self.bufs]
        if prepared:
            self.inp.t, self.inp.yw, self.inp.w = ptr
        else:
            self.inp.t, self.inp.y, self.inp.dy = ptr
        self.inp.n_points_total, self.inp.n_out_total = int(self.off[-1]), int(self.out_off[-1])

    def fill(self, seed):
        import torch
        rng = np.random.default_rng(seed)
        cols = [[], [], []]
        for i, (n, _) in enumerate(self.sizes):
            t = np.sort(rng.uniform(0, 900.0, n))
            y = np.sin(2 * np.pi * t / rng.uniform(1, 9)) + 0.1 * rng.standard_normal(n)
            dy = np.exp(rng.normal(-3, 0.3, n))
            if self.prepared:
                w = dy ** -2 / np.sum(dy ** -2)
                yw = w * (y - np.dot(w, y))
                c = self.cv[i]
                c.yy, c.ybar = float(np.dot(w, (y - np.dot(w, y)) ** 2)), 0.0
                y, dy = yw.astype(np.float32), w.astype(np.float32)
                c.yw_sum, c.w_sum = float(y.astype(float).sum()), float(dy.astype(float).sum())
            for col, v in zip(cols, (t, y, dy)):
                col.append(v)
        for b, col in zip(self.bufs, cols):
            b.copy_(torch.from_numpy(np.concatenate(col)))
        torch.cuda.synchronize()

    def launch(self, h, stream=None, best=False):
        from cuvarbase_gb300 import _lib
        L = _lib.load()
        a = ctypes.byref(self.inp)
        bk, bp = (x.data_ptr() for x in self.best)
        if self.prepared:
            rc = L.cuvgls_gls_best(h.ptr, a, bk, bp, stream) if best else \
                L.cuvgls_gls_batch(h.ptr, a, self.out.data_ptr(), stream)
        else:
            rc = L.cuvgls_gls_raw(h.ptr, a, None if best else self.out.data_ptr(),
                                  bk if best else None, bp if best else None, stream)
        h.check(rc, "several plans")

    def powers(self, h, stream=None):
        self.launch(h, stream)
        h.sync(stream, -1)
        return self.out.cpu().numpy()

    def alone(self, h):
        """The powers of each curve from a call of its own."""
        res = np.empty(int(self.out_off[-1]), np.float32)
        cv, n = self.inp.curves, self.inp.n_curves
        for i in range(n):
            self.inp.curves = ctypes.addressof(self.cv[i])
            self.inp.n_curves = 1
            q = slice(int(self.out_off[i]), int(self.out_off[i + 1]))
            res[q] = self.powers(h)[q]
        self.inp.curves, self.inp.n_curves = cv, n
        return res

    def check_best(self, want):
        """The best frequencies found are those of the powers `want`."""
        k, p = (x.cpu().numpy() for x in self.best)
        for i in range(len(self.sizes)):
            P = want[int(self.out_off[i]):int(self.out_off[i + 1])]
            assert P[k[i]] >= P.max() - TOL and abs(float(p[i]) - float(P.max())) <= TOL


@pytest.fixture(params=[-1.0, 2.0])
def h(request):
    from cuvarbase_gb300 import _lib
    hh = _lib.Handle(sigma=request.param, m=8)
    yield hh
    hh.close()


@pytest.mark.parametrize("prepared", [False, True])
def test_device_buffers(h, prepared):
    b = Batch(SIZES, 1, prepared)
    want = b.alone(h)
    assert np.abs(b.powers(h) - want).max() <= TOL
    b.launch(h, best=True)
    h.sync(None, -1)
    b.check_best(want)


@pytest.mark.parametrize("prepared", [False, True])
def test_two_streams_in_turn(h, prepared):
    """Calls on two streams without a wait in between: one arena, one set of
    side streams."""
    from cuvarbase_gb300 import _lib
    streams = [_lib.Stream(), _lib.Stream()]
    batches = [Batch(SIZES, 10 + k, prepared) for k in range(2)]
    want = [b.alone(h) for b in batches]
    for _ in range(5):
        for b in batches:
            b.out.fill_(-7.0)
        import torch
        torch.cuda.synchronize()
        for b, s in zip(batches, streams):
            b.launch(h, s.ptr)
        for s in streams:
            h.sync(s.ptr, -1)
        for b, w in zip(batches, want):
            assert np.abs(b.out.cpu().numpy() - w).max() <= TOL


@pytest.mark.parametrize("best", [False, True])
def test_captured_plan(h, best):
    """The side streams inside a captured plan, replayed on other data."""
    from cuvarbase_gb300 import _lib
    L = _lib.load()
    b = Batch(SIZES, 20)
    plan, s = ctypes.c_void_p(), _lib.Stream()
    bk, bp = (x.data_ptr() for x in b.best)
    h.check(L.cuvgls_gls_plan_create(h.ptr, ctypes.byref(b.inp), None if best else b.out.data_ptr(),
                                     bk if best else None, bp if best else None,
                                     ctypes.byref(plan)), "plan")
    try:
        for seed in (21, 22):
            b.fill(seed)
            want = b.alone(h)
            for _ in range(3):
                b.out.fill_(-7.0)
                import torch
                torch.cuda.synchronize()
                assert L.cuvgls_gls_plan_launch(plan, s.ptr) == 0
                h.sync(s.ptr, -1)
                if best:
                    b.check_best(want)
                else:
                    assert np.abs(b.out.cpu().numpy() - want).max() <= TOL
    finally:
        L.cuvgls_gls_plan_destroy(plan)


@pytest.mark.parametrize("warmed", [False, True])
def test_callers_own_capture(warmed):
    """A batch captured by the caller, on a handle whose side streams are there
    (warmed) and on one that has run batches of one plan only."""
    import torch
    from cuvarbase_gb300 import _lib
    h = _lib.Handle(sigma=2.0, m=8)
    try:
        b = Batch(SIZES, 30, prepared=True)
        st = torch.cuda.Stream()
        want = b.alone(h)                       # (tables of every plan)
        big = Batch([(3000, 120000)] * 40, 31, prepared=True)   # (and a large arena)
        big.powers(h)
        if warmed:
            h.check(_lib.load().cuvgls_warm(h.ptr, 500, 1000, 0), "warm")
        big.powers(h, st.cuda_stream)           # the handle's last stream
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st, capture_error_mode="relaxed"):
            b.launch(h, st.cuda_stream)
        for _ in range(3):
            b.out.fill_(-7.0)
            torch.cuda.synchronize()
            g.replay()
            torch.cuda.synchronize()
            assert np.abs(b.out.cpu().numpy() - want).max() <= TOL
    finally:
        h.close()


@pytest.mark.parametrize("prepared", [False, True])
@pytest.mark.parametrize("chunk_mb", [1, 16, 2048])
def test_small_workspaces(chunk_mb, prepared):
    """From the smallest workspace to one that holds everything (0.1 GB of
    records, 0.7 GB of intermediates): each plan by itself in several groups and
    chunks, shared preparation with one intermediate, and the plans beside each
    other all give the same powers."""
    from cuvarbase_gb300 import _lib
    sizes = [(n, nf) for nf in (700, 3000, 9000, 20000) for n in [400, 900, 3000] * 150]
    b = Batch(sizes, 40, prepared)
    want = None
    for mb in (2048, 512, 256, 160, 128, 96, 64, 40, 28, 20, 16):
        h = _lib.Handle(sigma=2.0, m=8, workspace_bytes=mb << 20, chunk_mb=chunk_mb)
        try:
            b.out.fill_(-7.0)
            got = b.powers(h)
        finally:
            h.close()
        want = got if want is None else want
        assert np.abs(got - want).max() <= TOL
    few = Batch(sizes[:3] + sizes[450:453], 41, prepared)
    h = _lib.Handle(sigma=2.0, m=8)
    try:
        assert np.abs(few.powers(h) - few.alone(h)).max() <= TOL
    finally:
        h.close()
