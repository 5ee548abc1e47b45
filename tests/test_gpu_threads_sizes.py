"""Calls of several threads whose kernels take shared memory by their sizes: a small
call between a large one's set-up and its launch must not lower the large one's limit
(the launch would be refused).  Straight C calls in tight loops, which run outside the
interpreter's lock."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _hammer(calls, n):
    import torch
    errors, start = [], threading.Barrier(len(calls))

    def work(call):
        with torch.cuda.stream(torch.cuda.Stream()):
            st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
            start.wait()
            for _ in range(n):
                if call(st):
                    errors.append(1)
            torch.cuda.current_stream().synchronize()
    threads = [threading.Thread(target=work, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors


def test_fan_projections_of_two_sizes(vg):
    """52 and 108 KB of line tables and sums, blocks of whole views."""
    import torch
    from vir_gb300 import _core, _lib
    L, na = _lib.load(), 700
    angs = np.linspace(0, 2 * np.pi, na, endpoint=False)
    x, out = torch.rand((4, 4), device="cuda"), {}
    xT, trig = x.t().contiguous(), _core.trig_cache.get(angs, np.float32, x.device)

    def fp(nu):
        g = _lib.DD2DGeom(4, 4, na, nu, _core.f32(20.0 / nu), 0.0, 1.0, 60.0, 100.0, 1, 0)
        o = out[nu] = torch.empty((na, nu), device="cuda")
        p = [ctypes.c_void_p(t.data_ptr()) for t in (x, xT, trig, o)]
        return lambda st: L.vg_dd2d_fp(ctypes.byref(g), *p, st)
    torch.cuda.synchronize()
    _hammer([fp(nu) for nu in (13312, 27648)], 4000)
    from vir_gb300.sys_mat import dd
    for nu, o in out.items():
        assert torch.equal(dd.dd_fp_fan_2d(x, angs, nu, 60.0, 100.0, du=20.0 / nu), o)


def test_row_filters_of_three_lengths(vg):
    """50, 100 and 200 KB of row buffers."""
    import torch
    from vir_gb300 import _core, _lib
    from vir_gb300.filtration import _device_spectrum, filter_rows_device
    L, rows = _lib.load(), [torch.rand((1, nu), device="cuda") for nu in (1500, 3000, 6000)]
    outs = [torch.empty_like(r) for r in rows]
    keep = []

    def run(r, o):
        z, spec, tw = _device_spectrum(r.shape[1], 1.0, "ramp", 0.5, True, r.device)
        keep.append((spec, tw))
        p = ctypes.c_void_p
        return lambda st: L.vg_filter_rows_fft(p(r.data_ptr()), 1, r.shape[1], z, p(spec.data_ptr()),
                                               p(tw.data_ptr()), None, p(o.data_ptr()), st)
    calls = [run(r, o) for r, o in zip(rows, outs)]
    torch.cuda.synchronize()
    _hammer(calls, 10000)
    for r, o in zip(rows, outs):
        assert torch.equal(filter_rows_device(r), o)
