"""The FDK back projection's column kernel where it changes form: one and two
pairs of slices per lane (slices up to 64, 65 to 128, just above 128), one
slice, views not a multiple of the table's 32 or the sums' 16, views whose
taps lie partly or wholly off the detector (a detector smaller than the
object, shifted off its axis, or one bin wide), and one-column images.

Tolerance: detector positions carry a few float32 roundings of at most 128
bins, 3e-5 bin, on steps between bins of up to twice the filtered values'
magnitude, and the filter's own float32 error is below 1e-5: 2e-4 of the
largest value against the FP64 oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# shape, na, nu, nv, du, dv, su, sv, DSO, DSD
CASES = {
    "one": ((9, 10, 1), 17, 40, 8, 0.8, 0.9, 0.0, 0.0, 40.0, 60.0),
    "pair": ((6, 17, 64), 33, 50, 128, 0.9, 1.0, 0.25, -0.5, 90.0, 140.0),
    "two": ((7, 8, 65), 48, 40, 110, 1.0, 1.1, 0.0, 0.0, 80.0, 120.0),
    "over": ((5, 3, 129), 31, 30, 128, 1.0, 1.7, 0.0, 0.0, 150.0, 230.0),
    "small": ((20, 21, 40), 40, 18, 20, 1.0, 1.0, 0.0, 0.0, 40.0, 60.0),
    "shifted": ((16, 16, 33), 64, 30, 30, 1.2, 1.2, 9.0, -11.0, 40.0, 60.0),
    "bin": ((3, 3, 70), 5, 1, 1, 4.0, 4.0, 0.0, 0.0, 40.0, 60.0),
    "column": ((1, 1, 100), 16, 9, 120, 0.5, 1.5, 0.0, 0.0, 100.0, 160.0),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_fdk_columns_vs_oracle(vg, orc, name):
    from vir_gb300 import reconstruction as rc
    shape, na, nu, nv, du, dv, su, sv, DSO, DSD = CASES[name]
    f32 = lambda v: float(np.float32(v))
    rng = np.random.default_rng(11)
    y = rng.random((na, nu, nv)).astype(np.float32)
    angs = np.linspace(0, 2 * np.pi, na, endpoint=False) + 0.1
    kw = dict(du=f32(du), dv=f32(dv), su=f32(su), sv=f32(sv))
    got = rc.fdk(y, angs, shape, DSO, DSD, **kw)
    ref = orc.fdk(y, angs, shape, DSO, DSD, **kw)
    assert np.abs(got - ref).max() <= 2e-4 * np.abs(ref).max()
