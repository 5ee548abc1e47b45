"""The pixel-driven FBP back projection at the sizes where its launch changes:
tiles of 16 x 32 pixels cut at their edges, 1 to 8 blocks of views per tile,
view blocks of 256, one-bin and one-pixel inputs, pixels off the detector.

Tolerance: a bin coordinate of up to nu / 2 = 200 carries three float32
roundings, 4e-5 bins, and filtered values here differ by at most 1 between
bins: 5e-5 of the largest value against the FP64 oracle."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fan", [False, True])
@pytest.mark.parametrize("shape,na,nu,su", [
    ((16, 32), 31, 40, 0.0),      # one tile, too few views to split
    ((17, 33), 64, 41, 0.25),     # split over 2 blocks
    ((5, 70), 300, 90, -0.5),     # over 8, ragged
    ((64, 40), 257, 1, 0.0),      # one bin; a view block of 256 and one more
    ((1, 1), 700, 9, 0.0),
    ((200, 170), 33, 401, 1.5),
])
def test_fbp_pixels_vs_oracle(vg, orc, fan, shape, na, nu, su):
    import torch
    from vir_gb300 import _core
    from vir_gb300.reconstruction import _geom
    rng = np.random.default_rng(3)
    q = rng.random((na, nu)).astype(np.float32)
    angs = np.linspace(0.1, 0.1 + 2 * np.pi, na, endpoint=False)
    f = lambda v: float(np.float32(v))
    DSO, DSD = (f(260.0), f(430.0)) if fan else (0.0, 0.0)
    du, d = f(0.9), f(0.8)
    qt = torch.from_numpy(q).cuda()
    trig = _core.trig_cache.get(angs, np.float32, qt.device)
    img = torch.full(shape, float("nan"), device="cuda")
    g = _geom(*shape, na, nu, du, su, d, DSO, DSD, int(fan))
    _core.call("vg_fbp2d_bp", ctypes.byref(g), _core.ptr(qt), _core.ptr(trig), _core.ptr(img),
               _core.stream(qt.device))
    ref = orc.fbp2d_bp(q, angs, shape, fan=fan, DSO=DSO, DSD=DSD, du=du, su=f(su), d_pix=d)
    assert np.abs(img.cpu().numpy() - ref).max() <= 5e-5 * np.abs(ref).max()


@pytest.mark.parametrize("na", [20, 40, 200, 700])
def test_infinite_bin_of_the_last_view(vg, na):
    """An infinite bin of the last view is infinity, not NaN, where only the interpolation
    towards it sees it, also where a tile's views are shared by several blocks (40 views and
    more): the sums of parts keep it as the sum in one block does."""
    import torch
    from vir_gb300 import _core, _lib
    nx, ny, nu, k = 40, 36, 64, 30
    g = _lib.DD2DGeom(nx, ny, na, nu, 1.0, 0.0, 1.0, 60.0, 110.0, 1, 0)
    trig = _core.trig_cache.get(np.linspace(0.1, 6.2, na), np.float32, torch.device("cuda", 0))

    def bp(q):
        out = torch.empty((nx, ny), device="cuda")
        _lib.call("vg_fbp2d_bp", ctypes.byref(g), q.data_ptr(), trig.data_ptr(), out.data_ptr(), _core.stream())
        return out

    def bin_of(j, value):
        q = torch.zeros((na, nu), device="cuda")
        q[na - 1, j] = value
        return bp(q)
    # pixels between bins k - 1 and k: reached from bin k, and not from k + 1
    want = (bin_of(k, 1.0) > 0) & ~(bin_of(k + 1, 1.0) > 0) & (bin_of(k - 1, 1.0) > 0)
    assert bool(want.any())
    assert bool(torch.isposinf(bin_of(k, float("inf")))[want].all())
