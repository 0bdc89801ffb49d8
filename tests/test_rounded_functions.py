"""gt_round.cuh (values rounded once without FP64 arithmetic) against numpy's double functions.

Where a function accepts its argument, its result is the correctly rounded one, which is also the
double result rounded to float: no tolerance.  It may decline (the caller then works in
double): 2 * 2^-38 / 2^-24 = 2^-13 of the calls to first order, 2^-12 at the lower end of a
binade; the limit below is 2^-11.
"""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "graptor_gb300", "csrc")
SRC = """
#include "gt_round.cuh"
extern "C" long run(int f, long n, const float *a, const float *b, float *out, unsigned char *ok) {
  for (long i = 0; i < n; ++i)
    ok[i] = f == 0 ? gt::cos_round(a[i], out[i]) : f == 1 ? gt::atan_round(a[i], out[i])
          : f == 2 ? gt::hyp_round(a[i], b[i], out[i]) : gt::cube_round(a[i], out[i]);
  return 0;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("round")
    (d / "r.cpp").write_text(SRC)
    so = str(d / "r.so")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, str(d / "r.cpp"),
                    "-o", so], check=True)
    return ctypes.CDLL(so)


def _edges(rng, n):
    """Arguments near multiples of pi/2, near k / 8 and k / 16 (the reductions' breaks), and tiny and huge ones."""
    step = rng.integers(-500, 500, n).astype(np.float32)
    return np.concatenate([
        np.float32(c) * (1 + step * np.float32(2.0 ** -23)) for c in
        (np.pi / 4, np.pi / 2, 3 * np.pi / 4, np.pi, 1 / 16, 3 / 16, 0.5, 15 / 16, 1.0, 16.0 / 15, 8.0)
    ] + [np.float32(10.0) ** rng.uniform(-44, 38, n).astype(np.float32)])


@pytest.mark.parametrize("f", ["cos", "atan", "hyp", "cube"])
def test_accepted_values_are_correctly_rounded(lib, f):
    rng = np.random.default_rng(5)
    n = 200000
    spread = (rng.uniform(-1, 1, n) * 2.0 ** rng.integers(-20, 20, n)).astype(np.float32)
    plain = rng.uniform(-3.9, 3.9, n).astype(np.float32)
    a = np.concatenate([plain, spread, _edges(rng, 2000), -_edges(rng, 2000)])
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan], np.float32)
    b = rng.permutation(a)
    a, b = np.concatenate([a, special]), np.concatenate([b, special[::-1]])
    out, ok = np.empty_like(a), np.zeros(a.size, np.uint8)
    P = ctypes.c_void_p
    lib.run(["cos", "atan", "hyp", "cube"].index(f), ctypes.c_long(a.size), a.ctypes.data_as(P),
            b.ctypes.data_as(P), out.ctypes.data_as(P), ok.ctypes.data_as(P))
    ok = ok.astype(bool)
    x, y = a.astype(np.float64), b.astype(np.float64)
    with np.errstate(all="ignore"):
        want = {"cos": lambda: np.cos(x), "atan": lambda: np.arctan(x), "hyp": lambda: np.sqrt(x * x + y * y),
                "cube": lambda: x * x * x}[f]().astype(np.float32)
    np.testing.assert_array_equal(out[ok], want[ok])
    assert (~ok[:n]).mean() <= 2.0 ** -11, (~ok[:n]).mean()
