"""CPU test of the Siddon walk's start (axis_start in vir_gb300/csrc/siddon2d.cu):
the device code itself, compiled for the host, against a search over all planes --
for start parameters inside the grid, on its planes, and outside it on both sides."""
import ctypes
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vir_gb300", "csrc", "siddon2d.cu")

HOST = r"""
#include <algorithm>
#include <cmath>
#include <cstring>
using std::fma; using std::max; using std::min;
#define __device__
#define __forceinline__ inline
static double d_mul(double a, double b) { return a * b; }
static double d_sub(double a, double b) { return a - b; }
static double __dmul_rn(double a, double b) { return a * b; }
static double __drcp_rn(double a) { return 1.0 / a; }
static double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
static long long __double_as_longlong(double a) { long long r; std::memcpy(&r, &a, 8); return r; }
static int __double2hiint(double a) { return (int)(__double_as_longlong(a) >> 32); }
static int __double2int_rd(double a) {
    a = std::floor(a);
    return a >= 2147483647.0 ? 2147483647 : a <= -2147483648.0 ? (int)-2147483648LL : (int)a;
}
struct SidGeom { double d_pix, inv_dpix; };
%s
extern "C" int start(double d_pix, int n, double o0, double d, double tb, double *t, double *all) {
    SidGeom g = {d_pix, 1.0 / d_pix};
    Axis a;
    axis_start(a, g, o0, d, rcp_of(d), n, tb, nullptr);
    for (int i = 0; i <= n; ++i) all[i] = cross_at(a, d_pix, i, nullptr);
    *t = a.t;
    return a.o == DONE ? -1 : a.i;
}
"""


@pytest.fixture(scope="module")
def start(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    src = open(SRC).read()
    part = lambda name, end: src[src.index(name):src.index(end, src.index(name))]
    code = "".join([
        part("__device__ __forceinline__ double edge(", "\n__device__ __forceinline__ double div_pix"),
        part("__device__ __forceinline__ double div_by(", "\nstruct Ray"),
        part("__device__ __forceinline__ long long ord64(", "\n// (float)h for h"),
    ])
    assert re.search(r"void axis_start\(", code)
    d = tmp_path_factory.mktemp("siddon")
    cpp, so = str(d / "start.cpp"), str(d / "start.so")
    with open(cpp, "w") as fh:
        fh.write(HOST % code)
    subprocess.run(["g++", "-O1", "-ffp-contract=off", "-shared", "-fPIC", "-o", so, cpp], check=True)
    L = ctypes.CDLL(so)
    dbl, vec = ctypes.c_double, np.ctypeslib.ndpointer(np.float64)
    L.start.argtypes = [dbl, ctypes.c_int, dbl, dbl, dbl, vec, vec]
    return L.start


@pytest.mark.parametrize("n,d_pix", [(1, 1.0), (2, 0.7), (16, 1.0), (97, 0.9)])
def test_axis_start_is_the_first_crossing_from_tb(start, n, d_pix):
    rng = np.random.default_rng(7)
    t, planes = np.zeros(1), np.zeros(n + 1)
    half = 0.5 * n * d_pix
    for d in list(rng.uniform(0.05, 1.0, 20)) + list(-rng.uniform(0.05, 1.0, 20)):
        o0 = rng.uniform(-half, half)
        on_plane = (d_pix * (rng.integers(0, n + 1, 6) - 0.5 * n) - o0) / d
        inside = (rng.uniform(-half, half, 6) - o0) / d
        # up to five pixels and far outside, before and after the grid
        outside = [(s * (half + k * d_pix) - o0) / d for s in (-1, 1) for k in (0.5, 1.5, 2.5, 5.0, 1e6, 1e12)]
        for tb in np.concatenate([on_plane, inside, outside]):
            i = start(d_pix, n, o0, d, tb, t, planes)
            walk = range(n + 1) if d > 0 else range(n, -1, -1)
            want = next((k for k in walk if planes[k] >= tb), -1)
            assert i == want, (d, o0, tb)
            if want >= 0:
                assert t[0] == planes[want]
