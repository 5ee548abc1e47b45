"""The Siddon projector's walk where its start and its steps can go wrong:
negative directions, views along the axes and the diagonals (ties of the two
axes' crossings, rays nearly along an axis), odd and one-pixel images, rays
that miss, a pixel size whose reciprocal is inexact, and an image whose plane
positions exceed the shared-memory table.

The single walk must give the oracle's voxel sequences and FP64 lengths
exactly.  The eight-part walk visits the same segments with lengths rounded to
float32: over an image of ones its sum is within 4 * 2^-24 of the FP64 length
(a rounding per length, one per part's compensated sum, one of their sum, one
in hand); the pair's inner products differ by float32 rounding of the two sums alone, 1e-6."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# shape, n_dets, d_det, d_pix, angles
STEP = np.linspace(0, 2 * np.pi, 16, endpoint=False)
CASES = {
    "turn": ((37, 50), 81, 0.9, 1.0, STEP),
    "inexact": ((64, 33), 70, 1.3, 0.7, STEP + 0.013),
    "dot": ((1, 1), 9, 0.25, 1.0, STEP),
    "row": ((1, 130), 40, 3.1, 0.8, STEP + 1e-9),
    "miss": ((16, 16), 90, 1.0, 1.0, STEP + 0.2),
    "untabled": ((1040, 1030), 33, 43.7, 1.0, STEP[:9] + 0.3),
    "coarse": ((24, 24), 5, 6.0, 1.0, STEP + np.pi / 16),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_walk_vs_oracle(vg, orc, name):
    import torch
    from vir_gb300 import _core
    from vir_gb300._lib import call
    from vir_gb300.sys_mat import fp_2d_par
    shape, nu, d_det, d_pix, angs = CASES[name]
    dev = torch.device("cuda")
    trig = _core.trig_cache.get(angs, None, dev)
    na = len(angs)
    cnt = torch.empty((na, nu), dtype=torch.int32, device=dev)
    h = torch.empty((na, nu), dtype=torch.int64, device=dev)
    ln = torch.empty((na, nu), dtype=torch.float64, device=dev)
    call("vg_siddon2d_trace", *shape, _core.ptr(trig), na, nu, d_det, d_pix, _core.ptr(cnt),
         _core.ptr(h), _core.ptr(ln), _core.stream(dev))
    cnt_o, h_o, len_o = orc.siddons_trace_2d(shape, angs, nu, d_det, d_pix)
    assert np.array_equal(cnt.cpu().numpy(), cnt_o)
    assert np.array_equal(h.cpu().numpy().view(np.uint64), h_o)
    assert np.array_equal(ln.cpu().numpy(), len_o)

    ones = fp_2d_par.siddons_fp_2d(np.ones(shape, np.float32), angs, nu, d_det=d_det, d_pix=d_pix)
    assert np.all(np.abs(ones - len_o) <= 4 * 2.0 ** -24 * len_o)

    rng = np.random.default_rng(7)
    x = rng.random(shape).astype(np.float32)
    y = rng.random((na, nu)).astype(np.float32)
    ax = fp_2d_par.siddons_fp_2d(x, angs, nu, d_det=d_det, d_pix=d_pix).astype(np.float64)
    aty = fp_2d_par.siddons_bp_2d(y, angs, shape, d_det=d_det, d_pix=d_pix).astype(np.float64)
    lhs, rhs = float((ax * y).sum()), float((x * aty).sum())
    assert abs(lhs - rhs) <= 1e-6 * abs(lhs)
