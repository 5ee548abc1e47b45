"""The SIRT calls leave their callers' tensors as they are: a prepared state, or
an object given a new sinogram, writes to a buffer of its own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GEO = dict(geom="fan", DSO=60.0, DSD=110.0, du=1.5)


@pytest.mark.parametrize("iters", [2, 4])
def test_sirt_calls_do_not_write_their_inputs(vg, iters):
    import torch
    from vir_gb300 import reconstruction as rc
    angs = np.linspace(0, 2 * np.pi, 20, endpoint=False)
    gen = torch.Generator().manual_seed(4)
    a, b = (torch.rand((20, 48), generator=gen).cuda() for _ in range(2))
    a0, b0 = a.clone(), b.clone()
    rc.prepared_sirt.clear()
    xa = rc.sirt_2d(a, angs, (32, 32), iters=iters, **GEO)
    xb = rc.sirt_2d(b, angs, (32, 32), iters=iters, **GEO)
    assert torch.equal(a, a0) and torch.equal(b, b0)
    assert torch.equal(rc.sirt_2d(a, angs, (32, 32), iters=iters, **GEO), xa)
    s = rc.SIRT2D(a, angs, (32, 32), **GEO)
    s.load_sino(b)
    assert torch.equal(a, a0)
    assert torch.equal(s.run(iters - 1), xb)
