"""The FFT row filter at the edges of its block plan: the smallest transforms,
both parities of log2 of the length, the longest (one block per SM), fewer and
more rows than one wave of blocks (blocks then filter several rows with one
twiddle table), with and without a row weight.

Tolerance: two transforms of log2 z <= 14 levels, each level a few roundings of
2^-24, on values that grow with the square root of the length while the
filtered row's largest does not fall: 5e-6 of the largest value against the
float64 FFT."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu, rows", [(2, 3), (3, 1000), (5, 7), (33, 2000), (129, 913),
                                      (700, 1), (1024, 1100), (4096, 160), (8192, 153)])
def test_fft_rows_vs_float64(vg, orc, nu, rows):
    import torch
    from vir_gb300 import filtration
    rng = np.random.default_rng(nu)
    x = rng.standard_normal((rows, nu)).astype(np.float32)
    w = rng.random(nu).astype(np.float32)
    xs, ws = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    for weight, src in ((None, x.astype(np.float64)), (ws, x.astype(np.float64) * w)):
        got = filtration.filter_rows_device(xs, 0.8, "hann", 0.5, row_weight=weight,
                                            method="fft").cpu().numpy()
        ref = orc.filter_sino(src, du=0.8, filter_type="hann", cutoff=0.5)
        assert np.abs(got - ref).max() <= 5e-6 * np.abs(ref).max()
