"""gt_fix.cuh (detector coordinates in fixed point) against exact rational arithmetic and
against the same coordinates computed in FP64: the fixed-point ones are no further off."""
import ctypes
import os
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "graptor_gb300", "csrc")
SRC = """
#include "gt_fix.cuh"
template <int FIX> static void at(long n, const double *o, const int *x0, const int *x, const int *y, long long *out) {
  const gt::FixAngle a = gt::fix_angle(gt::to_fix<FIX>(o[0]), gt::to_fix<FIX>(o[1]), gt::to_fix<FIX>(o[2]));
  for (long k = 0; k < n; ++k) {  // from x0 to x by steps
    gt::FixNum t = gt::fix_at(a, x0[k], y[k]);
    for (int q = x0[k]; q < x[k]; ++q) gt::fix_step(t, a);
    out[k] = t.hi;
  }
}
extern "C" int bits(long long t) { return gt::fix_bits(t); }
extern "C" void run(int fix, long n, const double *o, const int *x0, const int *x, const int *y, long long *out) {
  if (fix == 52) at<52>(n, o, x0, x, y, out);
  if (fix == 48) at<48>(n, o, x0, x, y, out);
  if (fix == 44) at<44>(n, o, x0, x, y, out);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("fix")
    (d / "f.cpp").write_text(SRC)
    so = str(d / "f.so")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, str(d / "f.cpp"),
                    "-o", so], check=True)
    return ctypes.CDLL(so)


def test_fraction_bits_hold_the_coordinate(lib):
    """t 2^FIX stays below 2^62 and the bits give out (0: FP64) beyond 2^18."""
    b = lambda t: lib.bits(ctypes.c_longlong(t))  # noqa: E731
    for e in range(1, 40):
        for t in (2 ** e - 1, 2 ** e):
            assert t * 2 ** b(t) < 2 ** 62
            assert (b(t) == 0) == (t >= 2 ** 18)


@pytest.mark.parametrize("N,nd", [(17, 19), (64, 64), (128, 128), (256, 256), (300, 423), (341, 341), (342, 342),
                                  (512, 512), (3, 1018), (2048, 2900), (3, 16378), (5461, 5462), (16384, 90000)])
def test_coordinates_are_no_further_off_than_in_fp64(lib, N, nd):
    rng = np.random.default_rng(N + nd)
    fix = lib.bits(ctypes.c_longlong(nd + 2 * N))
    n, P = 60, ctypes.c_void_p
    worst_fix = worst_64 = Fraction(0)
    for ang in np.concatenate([rng.uniform(0, np.pi, 12), np.deg2rad([20.0, 45.0, 89.9, 110.0, 160.0])]):
        X, Y = np.cos(ang), np.sin(ang)
        o = np.array([X, Y, (nd - 1.0) / 2 - X * ((N - 1) / 2.0) - Y * ((N - 1) / 2.0)])
        x = np.append(rng.integers(0, N, n - 1), N - 1).astype(np.int32)
        y = np.append(rng.integers(0, N, n - 1), N - 1).astype(np.int32)
        x0 = np.where(rng.random(n) < 0.5, x, np.maximum(x - 40, 0)).astype(np.int32)
        out = np.zeros(n, np.int64)
        lib.run(fix, ctypes.c_long(n), o.ctypes.data_as(P), x0.ctypes.data_as(P), x.ctypes.data_as(P), y.ctypes.data_as(P),
                out.ctypes.data_as(P))
        t64 = x * o[0] + y * o[1] + o[2]
        for k in range(n):
            exact = int(x[k]) * Fraction(o[0]) + int(y[k]) * Fraction(o[1]) + Fraction(o[2])
            err = abs(Fraction(int(out[k]), 2 ** fix) - exact)
            assert err <= Fraction(1, 2 ** (fix + 1)) + Fraction(int(x[k]) + int(y[k]) + 1, 2 ** (fix + 17))
            worst_fix, worst_64 = max(worst_fix, err), max(worst_64, abs(Fraction(float(t64[k])) - exact))
    assert worst_fix <= worst_64, (float(worst_fix), float(worst_64))
