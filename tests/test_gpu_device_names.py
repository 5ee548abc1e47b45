"""The objects' ``device`` argument takes what torch takes: a torch.device, with an
index or without, or its name."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DEVICES = ["cuda:0", "cuda", "torch.device('cuda')", "torch.device('cuda:0')"]


def _dev(name):
    import torch
    return eval(name, {"torch": torch}) if name.startswith("torch") else name


@pytest.mark.parametrize("name", DEVICES)
def test_device_argument(vg, name):
    from vir_gb300 import batched, reconstruction as rc
    from vir_gb300.sys_mat import siddon
    angs = np.linspace(0, 2 * np.pi, 12, endpoint=False)
    y = np.random.default_rng(2).random((12, 24)).astype(np.float32)
    kw = dict(geom="fan", DSO=60.0, DSD=110.0, du=1.5)
    ref = rc.SIRT2D(y, angs, (16, 16), **kw).run(2)
    got = rc.SIRT2D(y, angs, (16, 16), device=_dev(name), **kw).run(2)
    assert (got == ref).all()
    b = batched.BatchedSIRT2D([dict(sino=y, ang_arr=angs, img_shape=(16, 16), **kw)], device=_dev(name))
    b.capture(2)
    b.run(2)
    assert (b.images()[0] == ref).all()
    y3 = np.random.default_rng(3).random((12, 10, 8)).astype(np.float32)
    cone = [rc.SIRT3D(y3, angs, (6, 6, 6), 60.0, 110.0, **k).run(2) for k in ({}, dict(device=_dev(name)))]
    assert (cone[0] == cone[1]).all()
    src = np.array([[-20.0, 0.3, 0.2], [-20.0, 1.3, 0.2]])
    trg = np.array([[20.0, 0.1, -0.3], [20.0, -2.1, 1.3]])
    a, c = (siddon.siddons_device(src, trg, 8, 1.0, **k) for k in ({}, dict(device=_dev(name))))
    assert (a[0] == c[0]).all() and (a[1] == c[1]).all()
