"""Rounding of the cone pairs' slice and row positions on short tiles: they are
counted from the tile's middle.

One column of 5 slices in one wide u cell (FP), or one detector column (BP), so
that the u part is one factor of the whole profile along v or z, and profiles
normalised by their length show the positions' rounding alone.  Within 2.5 rows
that is at most 5e-8 of a row (float32's spacing there over sqrt(12)), and the
rounding of rows per output, 8e-8 at 1.5 outputs from the middle, 1.2e-7: 1.3e-7
on each of two edges with steps of 0.41 between values of 0.58 (uniform ones) is
1.3e-7 of the profile, and the normalisation and the sums add 1e-7.  4e-7 allowed;
counted from 40 rows off, positions would carry 1.1e-6 and profiles as much."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DSO, DSD = 60.0, 100.0


def _unit(a):
    return a / np.linalg.norm(a, axis=-1, keepdims=True)


@pytest.mark.parametrize("kind", ["dd", "sf"])
def test_short_profiles_rounding(vg, orc, kind):
    from vir_gb300.sys_mat import dd, sp
    fp, bp = (dd.dd_fp_cone_3d, dd.dd_bp_cone_3d) if kind == "dd" else (sp.sf_fp_cone_3d, sp.sf_bp_cone_3d)
    ofp, obp = ((orc.dd_fp_cone_3d, orc.dd_bp_cone_3d) if kind == "dd" else
                (orc.sf_fp_cone_3d, orc.sf_bp_cone_3d))
    rng = np.random.default_rng(41)
    e_fp, e_bp = [], []
    for k in range(24):
        f = lambda v: float(np.float32(v))
        ang = np.array([0.05 + 0.3 * k])
        kw = dict(du=16.0, dv=f(rng.uniform(1.4, 1.9)), su=0.0, sv=f(rng.uniform(-0.5, 0.5)), d_pix=1.0)
        vol = rng.random((1, 1, 5)).astype(np.float32)
        y = rng.random((1, 1, 6)).astype(np.float32)
        # the detector stays inside the slices' shadow, the slices inside the rows'
        e_fp.append(_unit(fp(vol, ang, 1, 4, DSO, DSD, **kw)) - _unit(ofp(vol, ang, 1, 4, DSO, DSD, **kw)))
        e_bp.append(_unit(bp(y, ang, (1, 1, 4), DSO, DSD, **kw)) - _unit(obp(y, ang, (1, 1, 4), DSO, DSD, **kw)))
    for e in (e_fp, e_bp):
        assert np.linalg.norm(np.stack(e)) <= 4e-7 * np.sqrt(len(e))


def test_output_just_below_a_slice_boundary(vg, orc):
    """A tile of one output that starts 2^-25 of a slice below slice nz / 2, which
    float32 rounds onto it."""
    from vir_gb300.sys_mat import dd
    vol = np.random.default_rng(3).random((1, 1, 160)).astype(np.float32)
    kw = dict(du=16.0, dv=float(np.float32(5.0 / 3.0)), su=0.0, sv=0.5 - 2.0**-25, d_pix=1.0)
    ref = orc.dd_fp_cone_3d(vol, np.array([0.0]), 1, 1, DSO, DSD, **kw)
    got = dd.dd_fp_cone_3d(vol, np.array([0.0]), 1, 1, DSO, DSD, **kw)
    assert np.abs(got - ref).max() <= 5e-5 * np.abs(ref).max()
