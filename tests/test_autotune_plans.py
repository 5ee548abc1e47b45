"""Which saved entries of the autotuner's cache a geometry reads (CPU: the timing is
replaced)."""
import json

import pytest

# nx, ny, na, nu, du, su, d_pix, DSO, DSD, fan
FAN = (64, 64, 60, 96, 1.2, 0.0, 0.9, 100.0, 200.0, 1)      # the tap form serves it
COARSE = (64, 64, 60, 96, 4.8, 0.0, 0.9, 100.0, 200.0, 1)   # its sizes, bins of 2.7 pixels: a tile
PAR = (64, 64, 60, 96, 1.2, 0.0, 0.9, 0.0, 0.0, 0)


@pytest.fixture
def tune(tmp_path, monkeypatch):
    import torch
    from vir_gb300 import _lib, autotune
    monkeypatch.setenv("VIR_GB300_AUTOTUNE", str(tmp_path / "autotune.json"))
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda dev=None: "a GPU")
    best = {}
    monkeypatch.setattr(autotune, "time_fp_variants", lambda g, dev, reps=3: best["t"])

    def run(geo, t, variant=0):
        best["t"] = t
        return autotune.best_fp_variant(_lib.DD2DGeom(*geo, variant), "cuda:0")
    run.path = tmp_path / "autotune.json"
    run.taps = _lib.load().vg_dd2d_fp_variants()
    run.old_key = lambda geo: (f"dd2d_fp|fan={geo[9]}|nx=64|ny=64|nu=96|na~64|a_GPU"
                               f"|lib={_lib.load().vg_version()}")
    return run


def test_entries_from_before_the_tap_form(tune):
    tune.path.write_text(json.dumps({tune.old_key(FAN): {"variant": 2, "ms": {}},
                                     tune.old_key(PAR): {"variant": 3, "ms": {}}}))
    assert tune(FAN, {2: 1.0, tune.taps: 0.5}) == tune.taps   # timed again
    assert tune(PAR, {1: 0.1}) == 3                           # still good
    assert tune(COARSE, {1: 0.1}) == 2


def test_one_size_two_geometries(tune):
    assert tune(COARSE, {1: 0.2, 4: 0.1, tune.taps: 0.3}) == 4
    assert tune(FAN, {4: 0.3, tune.taps: 0.2}) == tune.taps
    assert tune(COARSE, {}) == 4 and tune(FAN, {}) == tune.taps
    assert tune(FAN, {}, variant=2) == tune.taps              # the geometry's own variant is no part of it
