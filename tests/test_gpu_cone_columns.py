"""The cone DD pair's column kernels (u-overlaps into a row buffer, then
v-overlaps) at the sizes where they change form: 1, 2 or 3 groups of 32 outputs
per warp, 16-byte and 4-byte column loads, ragged tiles, columns of up to four
and of more overlapped cells, windows longer than a row buffer, a driving axis
that changes with every view, and tiles shared by a cluster of blocks.

Tolerance: the pair's float32 geometry is held to 5e-5 of the largest value
against the FP64 oracle everywhere else; the same here."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# shape, nu, nv, na, du, dv, d_pix, DSO, DSD
CASES = {
    # nz a multiple of 4 (16-byte loads in the FP), nv not (4-byte loads in the BP); nv = 97: 2 x 64
    "fp16_bp4": ((20, 17, 64), 37, 97, 9, 1.1, 1.3, 0.9, 60.0, 110.0),
    # the other way round; nv = 96: one group of 96 in the FP, nz = 65: 64 + 1 in the BP
    "fp4_bp16": ((17, 20, 65), 33, 96, 9, 1.2, 1.2, 0.8, 60.0, 110.0),
    # one group of 32 either way, sizes below a tile
    "small": ((5, 3, 31), 7, 30, 11, 1.0, 1.0, 1.0, 30.0, 50.0),
    # thin slices: a v cell overlaps up to 4 slices (FP groups of 32)
    "thin": ((12, 14, 90), 24, 40, 8, 0.9, 2.1, 0.5, 40.0, 70.0),
    # small v cells: a voxel overlaps up to 4 rows and columns (BP groups of 32), 33 slices
    "fine": ((13, 12, 33), 90, 130, 8, 0.5, 0.5, 0.9, 40.0, 70.0),
    # more than 4 detector columns per voxel, or rows than a buffer holds: per-voxel and per-cell paths
    "wide": ((10, 9, 40), 90, 60, 6, 0.25, 0.4, 1.0, 40.0, 70.0),
    "tall": ((9, 10, 300), 20, 24, 6, 1.5, 9.0, 0.5, 40.0, 70.0),
    # enough views for clusters of 2, 4 and 8 blocks on one tile
    "views64": ((8, 8, 12), 20, 18, 64, 1.0, 1.0, 1.0, 30.0, 50.0),
    "views300": ((9, 8, 40), 24, 60, 300, 1.0, 1.0, 1.0, 40.0, 60.0),
}


def _angles(na, order):
    a = np.linspace(0.03, 0.03 + 2 * np.pi, na, endpoint=False)
    return a if order == "circle" else a[np.random.default_rng(4).permutation(na)]


@pytest.mark.parametrize("order", ["circle", "shuffled"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_cone_columns_vs_oracle(vg, orc, name, order):
    from vir_gb300.sys_mat import dd
    shape, nu, nv, na, du, dv, d, DSO, DSD = CASES[name]
    rng = np.random.default_rng(17)
    angs = _angles(na, order)
    kw = dict(du=du, dv=dv, su=0.3, sv=-0.4, d_pix=d)
    vol = rng.random(shape).astype(np.float32)
    y = rng.random((na, nu, nv)).astype(np.float32)
    for got, ref in ((dd.dd_fp_cone_3d(vol, angs, nu, nv, DSO, DSD, **kw),
                      orc.dd_fp_cone_3d(vol, angs, nu, nv, DSO, DSD, **kw)),
                     (dd.dd_bp_cone_3d(y, angs, shape, DSO, DSD, **kw),
                      orc.dd_bp_cone_3d(y, angs, shape, DSO, DSD, **kw))):
        assert np.abs(got - ref).max() <= 5e-5 * np.abs(ref).max()


def test_cone_columns_unaligned_and_nonfinite(vg):
    """Inputs that start off a 16-byte boundary give the aligned call's values,
    and a NaN cell or voxel reaches no output two columns or rows away from
    what it overlaps."""
    import torch
    from vir_gb300.sys_mat import dd
    rng = np.random.default_rng(5)
    shape, nu, nv, na = (16, 16, 32), 40, 64, 6
    angs = np.linspace(0.1, 0.1 + 2 * np.pi, na, endpoint=False)
    kw = dict(du=1.0, dv=1.0, d_pix=1.0, su=0.0, sv=0.0)
    for call, size in ((lambda t: dd.dd_fp_cone_3d(t, angs, nu, nv, 60.0, 100.0, **kw), shape),
                       (lambda t: dd.dd_bp_cone_3d(t, angs, shape, 60.0, 100.0, **kw), (na, nu, nv))):
        a = torch.from_numpy(rng.random(size).astype(np.float32)).cuda()
        b = torch.empty(a.numel() + 1, device="cuda")[1:].view(size)
        b.copy_(a)
        ra, rb = call(a), call(b)
        assert torch.allclose(ra, rb, rtol=0, atol=2e-6 * ra.abs().max().item())
        hit = torch.zeros_like(a)
        hit.view(-1)[a.numel() // 2 + 7] = 1.0
        near = call(hit) != 0
        near = torch.nn.functional.max_pool3d(near.float()[None, None], 5, 1, 2)[0, 0] > 0
        if size == shape:  # neighbouring views are not neighbours in space
            near = call(hit) != 0
            near = torch.nn.functional.max_pool2d(near.float()[:, None], 5, 1, 2)[:, 0] > 0
        a.view(-1)[a.numel() // 2 + 7] = float("nan")
        assert not bool((torch.isnan(call(a)) & ~near).any())


# shape, nu, nv, na, du, dv, d_pix, DSO, DSD: u cells over many pixels and voxels over
# many detector columns (4 at a time), rows longer than a buffer (in pieces of 128), both,
# a detector that reaches the pole of the inverse edge map, one cell for everything
WIDE = {
    "u": ((40, 38, 33), 9, 40, 7, 12.0, 1.4, 1.0, 60.0, 100.0),
    "u_fine": ((9, 12, 64), 500, 70, 7, 0.1, 1.3, 1.0, 40.0, 70.0),
    "v": ((9, 8, 301), 21, 7, 7, 1.2, 33.0, 0.5, 60.0, 110.0),
    "v_fine": ((7, 9, 40), 24, 900, 5, 1.2, 0.09, 0.9, 40.0, 70.0),
    "uv": ((30, 28, 150), 5, 5, 9, 16.0, 41.0, 1.0, 60.0, 100.0),
    "uv_fine": ((6, 7, 9), 300, 400, 5, 0.11, 0.12, 1.0, 30.0, 55.0),
    "pole": ((20, 24, 10), 60, 30, 16, 5.0, 1.5, 1.0, 60.0, 100.0),
    "all": ((12, 10, 90), 1, 1, 8, 400.0, 4000.0, 1.0, 60.0, 100.0),
}


@pytest.mark.parametrize("name", sorted(WIDE))
def test_cone_columns_wide_vs_oracle(vg, orc, name):
    from vir_gb300.sys_mat import dd
    shape, nu, nv, na, du, dv, d, DSO, DSD = WIDE[name]
    rng = np.random.default_rng(19)
    angs = _angles(na, "shuffled")
    f = lambda v: float(np.float32(v))
    kw = dict(du=f(du), dv=f(dv), su=f(0.3), sv=f(-0.4), d_pix=f(d))
    vol = rng.random(shape).astype(np.float32)
    y = rng.random((na, nu, nv)).astype(np.float32)
    for got, ref in ((dd.dd_fp_cone_3d(vol, angs, nu, nv, DSO, DSD, **kw),
                      orc.dd_fp_cone_3d(vol, angs, nu, nv, DSO, DSD, **kw)),
                     (dd.dd_bp_cone_3d(y, angs, shape, DSO, DSD, **kw),
                      orc.dd_bp_cone_3d(y, angs, shape, DSO, DSD, **kw))):
        assert np.abs(got - ref).max() <= 5e-5 * np.abs(ref).max()


@pytest.mark.parametrize("name", ["u", "u_fine", "v", "uv"])
def test_cone_sirt_wide_vs_unfused(vg, name):
    """The SIRT epilogues of the wide kernels: two updates equal those put together from
    the projections, whose order of sums is the same (1e-5, as for the other geometries)."""
    import torch
    from vir_gb300 import reconstruction as rc
    from vir_gb300.sys_mat import dd
    shape, nu, nv, na, du, dv, d, DSO, DSD = WIDE[name]
    f = lambda v: float(np.float32(v))
    kw = dict(du=f(du), dv=f(dv), su=f(0.3), sv=f(-0.4), d_pix=f(d))
    angs = _angles(na, "circle")
    fp = lambda x: dd.dd_fp_cone_3d(x, angs, nu, nv, DSO, DSD, **kw)
    bp = lambda y: dd.dd_bp_cone_3d(y, angs, shape, DSO, DSD, **kw)
    vol = torch.rand(shape, generator=torch.Generator().manual_seed(8)).cuda()
    y = fp(vol)
    got = rc.SIRT3D(y, angs, shape, DSO, DSD, **kw).run(2)
    ws, wi = fp(torch.ones_like(vol)), bp(torch.ones_like(y))
    div = lambda a, w: torch.where(w != 0, a / w, a)
    x = torch.full(shape, float(np.float32(1e-5)), device="cuda")
    for _ in range(2):
        x = x + div(bp(div(y - fp(x), ws)), wi)
    near = wi > 1e-3 * wi.max()  # voxels beside the detector are divided by slivers
    assert (got - x).abs()[near].max() <= 1e-5 * x.abs()[near].max()


@pytest.mark.parametrize("nz,nv,dv", [(64, 30, 2.9), (33, 20, 5.0), (30, 90, 1.1)])
def test_cone_nonfinite_stays_within_a_row(vg, nz, nv, dv):
    """A voxel or cell that is not finite reaches no output more than one row, or one
    column, beside what it overlaps (1 and 2 groups of outputs, thin and thick slices)."""
    import torch
    from vir_gb300.sys_mat import dd
    shape, nu, na = (14, 16, nz), 24, 6
    angs = np.linspace(0.1, 0.1 + 2 * np.pi, na, endpoint=False)
    kw = dict(du=1.1, dv=dv, su=0.31, sv=0.17, d_pix=0.7)
    for call, size, rows in ((lambda t: dd.dd_fp_cone_3d(t, angs, nu, nv, 60.0, 100.0, **kw), shape, nz),
                             (lambda t: dd.dd_bp_cone_3d(t, angs, shape, 60.0, 100.0, **kw), (na, nu, nv), nv)):
        for z in (rows // 2,):  # away from the ends, where rows are read 4 at a time from the last
            near = torch.zeros(call(torch.zeros(size, device="cuda")).shape, dtype=torch.bool, device="cuda")
            for du in (-1, 0, 1):
                for dz in (-1, 0, 1):
                    x = torch.zeros(size, device="cuda")
                    if size == shape:
                        x[7, max(0, 9 + du) % 16, z + dz] = 1.0
                        near |= call(x) != 0
                        x.zero_()
                        x[7 + du, 9, z + dz] = 1.0
                    else:
                        x[2, 12 + du, z + dz] = 1.0
                    near |= call(x) != 0
            x = torch.rand(size, generator=torch.Generator().manual_seed(6)).cuda()
            x[(7, 9, z) if size == shape else (2, 12, z)] = float("inf")
            assert not bool((~torch.isfinite(call(x)) & ~near).any())
