"""The fan-beam forward projection's tap form (vg_dd2d_fp_variants' last
variant) and the back projection's view split, where they change form: bins
of up to 1, 2, 3 and more pixels, odd and one-line images, few views (bins of
a view over several blocks, lines over several warps), a detector near its
inverse map's pole (the exact share), whole views of more than 768 bins in the
SIRT epilogue, 1, 2 and 4 blocks of views per tile.

Tolerance: bin positions carry three float32 roundings of at most two image
widths, 7e-5 pixel for the sizes here, on pixel steps of at most 1: 1e-4 of the
largest value against the FP64 oracle, as for the integral form."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# shape, nu, na, du, su, d_pix, DSO, DSD
CASES = {
    "fine": ((65, 64), 190, 7, 0.4, 0.0, 1.0, 90.0, 170.0),      # bins of 0.2-0.5 pixel
    "mid": ((48, 53), 61, 33, 1.6, 0.25, 1.0, 60.0, 100.0),      # about 1; odd lines
    "wide": ((40, 40), 32, 70, 2.2, -0.5, 1.0, 34.0, 52.0),      # up to 3 and more near the edges
    "line": ((1, 37), 40, 130, 1.0, 0.0, 1.0, 60.0, 80.0),       # a single line or pixel row
    "pole": ((24, 24), 330, 9, 0.7, 0.0, 1.0, 90.0, 130.0),      # detector out to 0.89 DSD
    "tall": ((200, 9), 260, 3, 1.0, 0.0, 1.0, 220.0, 300.0),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_taps_vs_oracle(vg, orc, name):
    from vir_gb300 import _lib
    from vir_gb300.sys_mat import dd
    shape, nu, na, du, su, d, DSO, DSD = CASES[name]
    g = _lib.DD2DGeom(*shape, na, nu, du, su, d, DSO, DSD, 1)
    L = _lib.load()
    assert L.vg_dd2d_fp_default_variant(ctypes.byref(g)) == L.vg_dd2d_fp_variants()
    rng = np.random.default_rng(29)
    img = rng.random(shape).astype(np.float32)
    y = rng.random((na, nu)).astype(np.float32)
    angs = np.linspace(0, 2 * np.pi, na, endpoint=False) + 0.02
    kw = dict(du=du, su=su, d_pix=d)
    for got, ref in ((dd.dd_fp_fan_2d(img, angs, nu, DSO, DSD, **kw),
                      orc.dd_fp_fan_2d(img, angs, nu, DSO, DSD, **kw)),
                     (dd.dd_bp_fan_2d(y, angs, shape, DSO, DSD, **kw),
                      orc.dd_bp_fan_2d(y, angs, shape, DSO, DSD, **kw))):
        assert np.abs(got - ref).max() <= 1e-4 * np.abs(ref).max()


@pytest.mark.parametrize("nu", [96, 801])
def test_taps_sirt_epilogue_vs_oracle(vg, orc, nu):
    """Three SIRT updates: the residual and its back projection tables from the
    tap form's epilogue, with one block per view (2e-4 as the other SIRT tests)."""
    from vir_gb300 import reconstruction as rc
    rng = np.random.default_rng(31)
    shape, na, DSO, DSD = (45, 50), 66, 70.0, 120.0
    du = 110.0 / nu
    img = rng.random(shape).astype(np.float32)
    angs = np.linspace(0, 2 * np.pi, na, endpoint=False)
    fp = lambda x: orc.dd_fp_fan_2d(x, angs, nu, DSO, DSD, du=float(np.float32(du)))
    bp = lambda s: orc.dd_bp_fan_2d(s, angs, shape, DSO, DSD, du=float(np.float32(du)))
    y = fp(img).astype(np.float32)
    xo = orc.sirt(y, fp, bp, shape, iters=4)
    x = rc.sirt_2d(y, angs, shape, geom="fan", DSO=DSO, DSD=DSD, du=du, iters=4)
    assert np.abs(x - xo).max() <= 2e-4 * np.abs(xo).max()


def test_taps_nan_stays_near(vg):
    """A NaN pixel reaches only the bins within two of those it projects to."""
    import torch
    from vir_gb300.sys_mat import dd
    angs = np.linspace(0.1, 6.0, 8)
    x = torch.rand((40, 44), generator=torch.Generator().manual_seed(1)).cuda()
    hit = torch.zeros_like(x)
    hit[17, 21] = 1.0
    fp = lambda t: dd.dd_fp_fan_2d(t, angs, 90, 60.0, 100.0, du=1.0)
    near = torch.nn.functional.max_pool1d((fp(hit) != 0).float()[:, None], 5, 1, 2)[:, 0] > 0
    x[17, 21] = float("nan")
    assert not bool((torch.isnan(fp(x)) & ~near).any())


# shape, nu, na (first view at 45 degrees), du, d_pix, DSO, DSD, tolerance.  The share to
# first order in the bin's change of width (du <= 3e-3 of the source's distance from the
# detector's end).  "scan" and "fine": bins of 0.67 and 0.17 pixel seen from far, positions
# within 64 pixels: three roundings of 64 * 2^-24 pixel on steps of at most 1, averaged over
# 64 lines of independent rounding: 1.5e-6 of a value of half the lines; 1e-5 has six times that.
# "dot": the source within half a pixel of the corner of a 2 x 2 image, where the share's
# first order would turn at the next pixel edge; bins down to 4e-4 pixel, so three roundings
# of 2 * 2^-24 pixel are 9e-4 of a step: 2e-3.
FIRST_ORDER = {
    "scan": ((64, 61), 131, 24, 1.2, 0.9, 500.0, 1000.0, 1e-5),
    "fine": ((64, 64), 400, 16, 0.3, 0.9, 500.0, 1000.0, 1e-5),
    "dot": ((2, 2), 1600, 8, 0.0012, 1.0, 1.45, 2.2, 2e-3),
}


@pytest.mark.parametrize("name", sorted(FIRST_ORDER))
def test_taps_first_order_vs_oracle(vg, orc, name):
    from vir_gb300 import _lib
    from vir_gb300.sys_mat import dd
    shape, nu, na, du, d, DSO, DSD, tol = FIRST_ORDER[name]
    g = _lib.DD2DGeom(*shape, na, nu, du, 0.0, d, DSO, DSD, 1)
    L = _lib.load()
    assert L.vg_dd2d_fp_default_variant(ctypes.byref(g)) == L.vg_dd2d_fp_variants()
    assert du <= 3e-3 * (DSD - 0.5 * nu * du)
    img = np.random.default_rng(37).random(shape).astype(np.float32)
    angs = np.pi / 4 + np.linspace(0, 2 * np.pi, na, endpoint=False)
    f = lambda v: float(np.float32(v))
    got = dd.dd_fp_fan_2d(img, angs, nu, DSO, DSD, du=du, d_pix=d)
    ref = orc.dd_fp_fan_2d(img, angs, nu, f(DSO), f(DSD), du=f(du), d_pix=f(d))
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max()


@pytest.mark.parametrize("n,nu,du,DSO,DSD", [(64, 3000, 0.026, 45.5, 64.0), (16, 3000, 0.0105, 11.6, 20.0),
                                             (256, 4200, 0.1, 181.3, 256.0)])
def test_source_beside_the_image_keeps_the_integral_form(vg, n, nu, du, DSO, DSD):
    """Half widths within 1 % of DSO / sqrt(2): the call gives the integral form's bits."""
    import torch
    from vir_gb300 import _core, _lib
    from vir_gb300.sys_mat import dd
    angs = np.pi / 4 + np.linspace(0, 2 * np.pi, 8, endpoint=False)
    x = torch.rand((n, n), generator=torch.Generator().manual_seed(3)).cuda()
    xT, out = x.t().contiguous(), torch.empty((8, nu), device="cuda")
    f = _core.f32
    g = _lib.DD2DGeom(n, n, 8, nu, f(du), 0.0, 1.0, f(DSO), f(DSD), 1, 4)
    _lib.call("vg_dd2d_fp", ctypes.byref(g), _core.ptr(x), _core.ptr(xT),
              _core.ptr(_core.trig_cache.get(angs, np.float32, x.device)), _core.ptr(out), _core.stream(x.device))
    assert torch.equal(dd.dd_fp_fan_2d(x, angs, nu, DSO, DSD, du=du), out)


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("du", [0.05, 0.3, 1.2])
def test_taps_nonfinite_pixel_reaches_what_it_overlaps(vg, du, value):
    """A pixel that is not finite makes exactly the bins non-finite that a pixel of 1 in its
    place reaches (shares to first order and exact, bins of 0.04 to 0.9 pixel)."""
    import torch
    from vir_gb300.sys_mat import dd
    shape, DSO, DSD = (40, 37), 60.0, 90.0
    nu = int(60 * DSD / DSO / du)
    angs = np.pi / 4 + np.linspace(0, 2 * np.pi, 12, endpoint=False)
    fp = lambda t: dd.dd_fp_fan_2d(t, angs, nu, DSO, DSD, du=du, su=0.31, d_pix=0.9)
    for at in ((17, 21), (0, 36), (39, 1)):
        x = torch.zeros(shape, device="cuda")
        x[at] = 1.0
        near = fp(x) != 0
        x = torch.rand(shape, generator=torch.Generator().manual_seed(6)).cuda()
        x[at] = value
        assert torch.equal(~torch.isfinite(fp(x)), near)
