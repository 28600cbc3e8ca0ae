"""The flutter kernel's mixed-precision offset (csrc/fvx_parts.cuh), compiled for the
host: wherever diff_f32 answers, its float is that of the rounded FP64
difference, and it answers for all but a few pairs."""
import ctypes
import shutil
import subprocess

import numpy as np
import pytest

from tests.test_x3_host import CSRC

SHIM = r'''
#include "fvx_parts.cuh"
using namespace fvx;
extern "C" void parts(int n, const double* x, float* out) {
  for (int i = 0; i < n; ++i) {
    const Parts p = split_f32(x[i]);
    out[3 * i] = p.h, out[3 * i + 1] = p.l, out[3 * i + 2] = p.r;
  }
}
extern "C" void diff(int n, const double* x, const double* y, float* out, unsigned char* same) {
  for (int i = 0; i < n; ++i) {
    bool s = true;
    out[i] = diff_f32(split_f32(x[i]), split_f32(y[i]), s);
    same[i] = s;
  }
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    d = tmp_path_factory.mktemp("parts")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC,
                    "-o", str(d / "shim.so"), str(d / "shim.cpp")], check=True)
    return ctypes.CDLL(str(d / "shim.so"))


def _ptr(a):
    return ctypes.c_void_p(a.ctypes.data)


def _pairs(kind, n=400000):
    rng = np.random.default_rng(23)
    f32, f64 = np.float32, np.float64
    x, y = rng.uniform(-20, 20, n), rng.uniform(-20, 20, n)
    if kind == "near":
        y = x + rng.standard_normal(n) * 2.0 ** -rng.integers(0, 50, n)
    elif kind == "ties":
        f = (x - y).astype(f32)
        mid = 0.5 * (f.astype(f64) + np.nextafter(f, f32(np.inf)))
        y = np.nextafter(x - mid, np.where(rng.random(n) < 0.5, np.inf, -np.inf))
    elif kind == "floats":
        x = x.astype(f32).astype(f64)
        y = x * (1.0 + 2.0 ** -rng.integers(8, 52, n).astype(f64))
    elif kind == "equal":
        y = x.copy()
    elif kind == "scales":
        s = 2.0 ** rng.integers(-40, 60, n).astype(f64)
        x, y = x * s, y * s * 2.0 ** -rng.integers(0, 40, n).astype(f64)
    elif kind == "not finite":
        x[::3], y[1::3] = np.nan, np.inf
        x[2::3] = -np.inf
    return x, y


@pytest.mark.parametrize("kind", ["apart", "near", "ties", "floats", "equal", "scales",
                                  "not finite"])
def test_difference_is_the_rounded_fp64_difference(lib, kind):
    x, y = _pairs(kind)
    out, same = np.empty(x.size, np.float32), np.empty(x.size, np.uint8)
    lib.diff(x.size, _ptr(x), _ptr(y), _ptr(out), _ptr(same))
    same = same.astype(bool)
    assert np.array_equal(out[same], (x - y).astype(np.float32)[same])
    if kind in ("apart", "equal"):
        assert same.mean() > 0.9999
    if kind == "not finite":
        assert not same.any()


@pytest.mark.parametrize("kind", ["apart", "near", "scales"])
def test_parts_are_exact(lib, kind):
    x = np.concatenate(_pairs(kind))
    out = np.empty((x.size, 3), np.float32)
    lib.parts(x.size, _ptr(x), _ptr(out))
    assert np.array_equal(out.astype(np.float64).sum(1), x)
