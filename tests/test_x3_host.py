"""The three-float cores of the FP64 particle sweeps (csrc/fvx_x3.cuh), compiled
for the host, against 40-digit arithmetic: f, f'/r and f'/r r^2 + 2 f over
r / sigma from 1e-9 to 1e6, both sides of every change of method, and the ends of
the range that the kernel admits.

Bounds.  The three floats carry 72 bits and every operation drops terms below
2^-66; with some twenty operations in a row 2^-60 is theirs.  The Gaussian
core's polynomials keep two floats from the second power on and one from the
sixth, whose terms are below 2^-9 and 2^-35 of the value: 2^-56.  FP64 rounding
of the result adds 2^-53."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

mp = pytest.importorskip("mpmath").mp
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "fluxvortex_gb300", "csrc")
SHIM = r'''
#include "fvx_x3.cuh"
#include "fvx_core_table.cuh"
using namespace fvx::x3;
static const float T[] = {FVX_CORE_TABLE};
extern "C" void cores(int gauss, int n, const double* t, const double* s, const double* sigma,
                      double* d, float* parts, double* out) {
  for (int i = 0; i < n; ++i) {
    F3 x[3], v[3];
    for (int k = 0; k < 3; ++k) {
      x[k] = diff(split(t[3 * i + k]), split(s[3 * i + k]));
      d[3 * i + k] = to_double(x[k]);
    }
    if (gauss)
      gaussian<true, true>(x[0], x[1], x[2], gaussian_core(sigma[i]), kCoreEnd, kCoreRows,
                           [](int row, int k) {
                             Row r;
                             for (int j = 0; j < kRowFloats; ++j)
                               r.c[j] = T[(2 * row + k) * kRowFloats + j];
                             return r;
                           },
                           v[0], v[1], v[2]);
    else
      winckelmans<true, true>(x[0], x[1], x[2], winckelmans_core(sigma[i]), v[0], v[1], v[2]);
    for (int k = 0; k < 3; ++k) {
      parts[9 * i + 3 * k] = v[k].h;
      parts[9 * i + 3 * k + 1] = v[k].m;
      parts[9 * i + 3 * k + 2] = v[k].l;
      out[3 * i + k] = to_double(v[k]);
    }
  }
}
'''


@pytest.fixture(scope="module")
def cores(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("x3")
    (d / "shim.cpp").write_text(SHIM)
    lib = str(d / "shim.so")
    subprocess.run([gxx, "-O1", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC,
                    "-o", lib, str(d / "shim.cpp"), "-lm"], check=True)
    fn = ctypes.CDLL(lib).cores
    P = ctypes.c_void_p

    def run(gauss, t, s, sigma):
        n = sigma.size
        d_, parts = np.empty((n, 3)), np.empty((n, 3, 3), np.float32)
        out = np.empty((n, 3))
        fn(int(gauss), n, *(P(a.ctypes.data) for a in (t, s, sigma, d_, parts, out)))
        return d_, parts, out

    return run


def _exact(gauss, t, s, sigma):
    """f, f'/r, their isotropic sum and that sum's scale."""
    d = [mp.mpf(float(a)) - mp.mpf(float(b)) for a, b in zip(t, s)]
    r2 = sum(x * x for x in d)
    sg = mp.mpf(float(sigma))
    if not gauss:
        q = r2 + sg * sg
        f = (r2 + mp.mpf(5) / 2 * sg * sg) / q ** mp.mpf(2.5)
        p = -(3 * r2 + mp.mpf(21) / 2 * sg * sg) / q ** mp.mpf(3.5)
    else:
        x = r2 / sg ** 2
        c = mp.sqrt(2 / mp.pi)
        if x < mp.mpf(1) / 4:
            a = [(-1) ** k / (mp.mpf(2) ** k * mp.factorial(k) * (2 * k + 3)) for k in range(25)]
            F = c * sum(v * x ** k for k, v in enumerate(a))
            G = 2 * c * sum(k * v * x ** (k - 1) for k, v in enumerate(a) if k)
        else:
            rho = mp.sqrt(x)
            e = mp.exp(-x / 2)
            g = mp.erf(rho / mp.sqrt(2)) - c * rho * e
            F, G = g / rho ** 3, (c * rho ** 3 * e - 3 * g) / rho ** 5
        f, p = F / sg ** 3, G / sg ** 5
    return [f, p, p * r2 + 2 * f], [abs(f), abs(p), 2 * f + abs(p) * r2]


@pytest.mark.parametrize("gauss", [False, True])
@pytest.mark.parametrize("kind", ["wake", "self", "edges", "small", "large"])
def test_cores_against_40_digits(cores, gauss, kind):
    mp.dps = 40
    rng = np.random.default_rng(len(kind))
    n = 150
    sigma = 0.5 * 2.0 ** -rng.uniform(0, 6, n)
    span = {"small": 1e-3, "large": 8000.0}.get(kind, 20.0)
    if kind == "small":
        sigma = 2.0 ** -rng.uniform(12, 22, n)
    elif kind == "large":
        sigma = 2.0 ** rng.uniform(0, 12.9, n)
    rho = 10.0 ** rng.uniform(-3, 3, n)
    if kind == "self":
        rho = 10.0 ** rng.uniform(-9, -1, n)
        rho[:5] = 0.0
    elif kind == "edges":   # interval ends, the singular core's start, powers of four
        x = np.concatenate([np.arange(0.25, 3.0, 0.25), [89.75, 90.0, 90.25, 128, 256, 1024, 4096]])
        rho = np.sqrt(np.resize(x, n) * (1.0 + rng.choice([-1e-7, 0, 1e-7, 1e-15, -1e-15], n)))
    t = rng.uniform(-span, span, (n, 3))
    u = rng.standard_normal((n, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    s = np.clip(t + np.minimum(rho * sigma, span)[:, None] * u, -8191.0, 8191.0)
    if kind == "self":
        s[:5] = t[:5]
    d, parts, out = cores(gauss, t, s, sigma)
    assert np.array_equal(d, t - s)                 # the FP64 difference, bit for bit
    bound = mp.mpf(2) ** (-56 if gauss else -60)
    for i in range(n):
        ref, scale = _exact(gauss, t[i], s[i], sigma[i])
        for k in range(3):
            got = sum(mp.mpf(float(v)) for v in parts[i, k])
            assert abs(got - ref[k]) <= bound * scale[k], (i, k, float(abs(got - ref[k]) / scale[k]))
            # to the nearest FP64 number (a tie's distance and the sum's own place)
            assert abs(mp.mpf(float(out[i, k])) - got) <= mp.mpf(2) ** -52.99 * abs(got), (i, k)
