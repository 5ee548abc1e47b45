"""The cone SF pair's column kernels at the sizes where they change form: 1, 2 or
3 groups of 32 outputs per warp, 16-byte and 4-byte loads, ragged tiles, columns
over more than 4 u cells, lines of more than 32 columns under 8 u cells, windows
longer than a row buffer, tiles shared by a cluster of blocks.

Tolerance: the pair is held to 5e-5 of the largest value against the FP64 oracle
elsewhere; the same here."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# shape, nu, nv, na, du, dv, d_pix, DSO, DSD
CASES = {
    "fp16_bp4": ((12, 9, 64), 21, 97, 5, 1.1, 1.3, 0.9, 40.0, 70.0),
    "fp4_bp16": ((9, 12, 65), 17, 96, 5, 1.2, 1.2, 0.8, 40.0, 70.0),
    "small": ((5, 3, 31), 7, 30, 7, 1.0, 1.0, 1.0, 30.0, 50.0),
    "thin": ((8, 9, 70), 14, 40, 5, 0.9, 2.1, 0.5, 40.0, 70.0),
    "wide_bp": ((7, 8, 33), 60, 50, 4, 0.3, 0.5, 1.0, 30.0, 55.0),
    "wide_fp": ((40, 44, 6), 9, 12, 4, 11.0, 2.0, 1.0, 60.0, 100.0),
    "tall": ((6, 7, 200), 12, 20, 4, 1.5, 8.0, 0.5, 40.0, 70.0),
    "views": ((8, 8, 12), 14, 12, 130, 1.0, 1.5, 1.0, 30.0, 50.0),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_sf_cone_columns_vs_oracle(vg, orc, name):
    from vir_gb300.sys_mat import sp
    shape, nu, nv, na, du, dv, d, DSO, DSD = CASES[name]
    rng = np.random.default_rng(23)
    angs = np.linspace(0.03, 0.03 + 2 * np.pi, na, endpoint=False)
    f = lambda v: float(np.float32(v))
    kw = dict(du=f(du), dv=f(dv), su=f(0.3), sv=f(-0.4), d_pix=f(d))
    vol = rng.random(shape).astype(np.float32)
    y = rng.random((na, nu, nv)).astype(np.float32)
    for got, ref in ((sp.sf_fp_cone_3d(vol, angs, nu, nv, DSO, DSD, **kw),
                      orc.sf_fp_cone_3d(vol, angs, nu, nv, DSO, DSD, **kw)),
                     (sp.sf_bp_cone_3d(y, angs, shape, DSO, DSD, **kw),
                      orc.sf_bp_cone_3d(y, angs, shape, DSO, DSD, **kw))):
        assert np.abs(got - ref).max() <= 5e-5 * np.abs(ref).max()


# Last tiles of 1, 2, 5 and 6 columns (pairs without a live column), the same with
# columns beside the detector, and magnifications of 1.4 to 3.5 in one tile, so that
# columns over 5 and 6 u cells (per-voxel path) lie between narrower ones.
PAIRS = {
    "one": ((9, 7, 40), 40, 44, 21, 1.0, 1.0, 40.0, 70.0),
    "two": ((10, 9, 70), 40, 64, 21, 1.0, 1.0, 40.0, 70.0),
    "five": ((13, 8, 33), 45, 41, 21, 1.0, 1.0, 40.0, 70.0),
    "six": ((14, 9, 66), 45, 72, 21, 1.0, 1.0, 40.0, 70.0),
    "beside": ((21, 22, 34), 12, 40, 33, 1.0, 1.0, 40.0, 70.0),
    "near": ((14, 13, 36), 60, 90, 33, 1.0, 1.2, 14.0, 28.0),
}


@pytest.mark.parametrize("name", sorted(PAIRS))
def test_sf_bp_pairs_skipped_vs_oracle(vg, orc, name):
    """Pairs of columns that use no row buffer, between and after ones that do."""
    from vir_gb300.sys_mat import sp
    shape, nu, nv, na, du, dv, DSO, DSD = PAIRS[name]
    angs = np.linspace(0.05, 0.05 + 2 * np.pi, na, endpoint=False)
    f = lambda v: float(np.float32(v))
    kw = dict(du=f(du), dv=f(dv), su=0.25, sv=0.5, d_pix=1.0)
    y = np.random.default_rng(29).random((na, nu, nv)).astype(np.float32)
    ref = orc.sf_bp_cone_3d(y, angs, shape, DSO, DSD, **kw)
    for _ in range(3):
        got = sp.sf_bp_cone_3d(y, angs, shape, DSO, DSD, **kw)
        assert np.abs(got - ref).max() <= 5e-5 * np.abs(ref).max()


def test_sf_cone_columns_nan_stays_near(vg):
    """A NaN voxel or cell reaches only outputs within two of those it overlaps."""
    import torch
    from vir_gb300.sys_mat import sp
    shape, nu, nv, na = (16, 16, 32), 40, 64, 6
    angs = np.linspace(0.1, 0.1 + 2 * np.pi, na, endpoint=False)
    kw = dict(du=1.0, dv=1.0, d_pix=1.0)
    for call, size in ((lambda t: sp.sf_fp_cone_3d(t, angs, nu, nv, 60.0, 100.0, **kw), shape),
                       (lambda t: sp.sf_bp_cone_3d(t, angs, shape, 60.0, 100.0, **kw), (na, nu, nv))):
        a = torch.rand(size, generator=torch.Generator().manual_seed(2)).cuda()
        hit = torch.zeros_like(a)
        hit.view(-1)[a.numel() // 2 + 7] = 1.0
        near = (call(hit) != 0).float()
        near = (torch.nn.functional.max_pool2d(near[:, None], 5, 1, 2)[:, 0] if size == shape
                else torch.nn.functional.max_pool3d(near[None, None], 5, 1, 2)[0, 0]) > 0
        a.view(-1)[a.numel() // 2 + 7] = float("nan")
        assert not bool((torch.isnan(call(a)) & ~near).any())


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("nz,nv,du", [(32, 64, 1.0), (70, 63, 1.0), (40, 90, 0.45)])
def test_sf_bp_nonfinite_cell_reaches_what_it_overlaps(vg, nz, nv, du, value):
    """A cell that is not finite makes exactly the voxels non-finite that a
    cell of 1 in its place reaches (1 and 2 groups of slices, 4- and 16-byte
    loads, columns over up to and over more than 4 u cells)."""
    import torch
    from vir_gb300.sys_mat import sp
    shape, nu, na = (13, 16, nz), 40, 6
    angs = np.linspace(0.1, 0.1 + 2 * np.pi, na, endpoint=False)
    bp = lambda t: sp.sf_bp_cone_3d(t, angs, shape, 60.0, 100.0, du=du, dv=1.03, su=0.31, sv=0.17, d_pix=1.0)
    for at in ((1, 20, nv // 2), (4, 13, 2), (3, 0, nv - 1)):
        y = torch.zeros((na, nu, nv), device="cuda")
        y[at] = 1.0
        near = bp(y) != 0
        y = torch.rand((na, nu, nv), generator=torch.Generator().manual_seed(6)).cuda()
        y[at] = value
        assert torch.equal(~torch.isfinite(bp(y)), near)


# shape, nu, nv, na, du, dv, d_pix, DSO, DSD: lines of more than 32 and 64 columns under 8
# u cells, v cells over 4 to 40 slices (pieces of 240 rows), both, one cell for everything,
# a detector that reaches the pole of the inverse edge map
FP_WIDE = {
    "u": ((90, 80, 20), 9, 30, 5, 18.0, 1.5, 1.0, 100.0, 160.0),
    "v4": ((9, 8, 160), 21, 33, 7, 1.2, 4.4, 0.5, 60.0, 110.0),
    "v40": ((8, 10, 500), 20, 9, 5, 1.2, 40.0, 0.5, 60.0, 110.0),
    "uv": ((40, 36, 250), 7, 5, 6, 17.0, 60.0, 1.0, 60.0, 100.0),
    "all": ((12, 10, 90), 1, 1, 8, 400.0, 4000.0, 1.0, 60.0, 100.0),
    "pole": ((40, 36, 10), 60, 30, 16, 5.0, 1.5, 1.0, 60.0, 100.0),
}


@pytest.mark.parametrize("name", sorted(FP_WIDE))
def test_sf_fp_wide_vs_oracle(vg, orc, name):
    from vir_gb300.sys_mat import sp
    shape, nu, nv, na, du, dv, d, DSO, DSD = FP_WIDE[name]
    angs = np.linspace(0.03, 0.03 + 2 * np.pi, na, endpoint=False)
    f = lambda v: float(np.float32(v))
    kw = dict(du=f(du), dv=f(dv), su=f(0.3), sv=f(-0.4), d_pix=f(d))
    vol = np.random.default_rng(31).random(shape).astype(np.float32)
    got = sp.sf_fp_cone_3d(vol, angs, nu, nv, DSO, DSD, **kw)
    ref = orc.sf_fp_cone_3d(vol, angs, nu, nv, DSO, DSD, **kw)
    assert np.abs(got - ref).max() <= 5e-5 * np.abs(ref).max()


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("nz,nv,dv", [(160, 13, 13.3), (160, 300, 0.31), (61, 70, 1.13), (64, 30, 2.9)])
def test_sf_fp_nonfinite_voxel_reaches_what_it_overlaps(vg, nz, nv, dv, value):
    """A voxel that is not finite makes exactly the cells non-finite that a voxel of 1 in
    its place reaches (running sums, 3 and 1 groups of v cells, 4- and 16-byte loads)."""
    import torch
    from vir_gb300.sys_mat import sp
    shape, nu, na = (14, 16, nz), 24, 6
    angs = np.linspace(0.1, 0.1 + 2 * np.pi, na, endpoint=False)
    fp = lambda t: sp.sf_fp_cone_3d(t, angs, nu, nv, 60.0, 100.0, du=1.1, dv=dv, su=0.31, sv=0.17, d_pix=0.7)
    for at in ((3, 9, nz // 2), (13, 0, 1), (7, 7, nz - 2)):
        x = torch.zeros(shape, device="cuda")
        x[at] = 1.0
        near = fp(x) != 0
        x = torch.rand(shape, generator=torch.Generator().manual_seed(6)).cuda()
        x[at] = value
        assert torch.equal(~torch.isfinite(fp(x)), near)


# shape, nu, nv, na, du, dv, d_pix, DSO, DSD: columns over more than 4 and more than 32 u
# cells, slices over 4 to 30 v cells (pieces of 480), both, more slices than a warp's 32
BP_WIDE = {
    "u": ((11, 9, 33), 120, 50, 7, 0.2, 1.2, 1.0, 40.0, 70.0),
    "u40": ((7, 6, 20), 500, 30, 5, 0.04, 1.2, 0.9, 30.0, 55.0),
    "v": ((9, 10, 64), 26, 500, 7, 1.1, 0.3, 1.0, 40.0, 70.0),
    "v30": ((6, 7, 40), 20, 2500, 5, 1.2, 0.06, 0.9, 40.0, 70.0),
    "uv": ((8, 5, 37), 90, 300, 40, 0.25, 0.3, 1.0, 40.0, 70.0),
    "beside": ((16, 17, 40), 30, 100, 20, 0.25, 0.3, 1.0, 40.0, 70.0),
}


@pytest.mark.parametrize("name", sorted(BP_WIDE))
def test_sf_bp_wide_vs_oracle(vg, orc, name):
    from vir_gb300.sys_mat import sp
    shape, nu, nv, na, du, dv, d, DSO, DSD = BP_WIDE[name]
    angs = np.linspace(0.03, 0.03 + 2 * np.pi, na, endpoint=False)
    f = lambda v: float(np.float32(v))
    kw = dict(du=f(du), dv=f(dv), su=f(0.3), sv=f(-0.4), d_pix=f(d))
    y = np.random.default_rng(31).random((na, nu, nv)).astype(np.float32)
    got = sp.sf_bp_cone_3d(y, angs, shape, DSO, DSD, **kw)
    ref = orc.sf_bp_cone_3d(y, angs, shape, DSO, DSD, **kw)
    assert np.abs(got - ref).max() <= 5e-5 * np.abs(ref).max()
