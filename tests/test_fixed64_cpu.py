"""The FP64 step's 64-bit fixed-point forms (csrc/pfa_fixed64.cuh), compiled for
the host, against the expressions they stand for in extended precision."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import PKG_DIR

SOURCE = r"""
#include <cstdint>
#include "pfa_fixed64.cuh"
using namespace pfa;
using namespace pfa::dev;

static uint64_t f63(double v) { return uint64_t(v * 0x1p63); }  // v in [0, 1]: exact to 2^-63

extern "C" int solve(int kind, double x, double y, double d, double l, double* g) {
  int64_t h1 = 0, h2 = 0;
  const bool ok = kind == 1   ? solve_fixed<1>(f63(x), f63(y), f63(d), f63(l), h1, h2)
                  : kind == 2 ? solve_fixed<2>(f63(x), f63(y), f63(d), f63(l), h1, h2)
                              : solve_fixed<3>(f63(x), f63(y), f63(d), f63(l), h1, h2);
  g[0] = h1 * 0x1p-60;
  g[1] = h2 * 0x1p-60;
  return ok;
}

extern "C" int sum_of_faces(int64_t n, int64_t s, int64_t e, int64_t w, int64_t* t) { return face_sum(n, s, e, w, *t); }

extern "C" void ranges(int64_t* r) {
  const Range60 v[3] = {kRangeFaces, kRangeCorners, kRangeFlux};
  for (int k = 0; k < 3; k++) {
    r[2 * k] = v[k].low;
    r[2 * k + 1] = v[k].most;
  }
}

// x^gamma from the monomials, in long double
extern "C" void exact(double x, double y, double d, double l, double* g) {
  typedef long double T;
  auto p = [](T v) { return v * v * v * (6 * v * v - 15 * v + 10); };
  const T pD = p(d), pL = p(l), pG = 1 - pD - pL;
  const T mono[6] = {pD * pD, pD * pG, pD * pL, pG * pG, pG * pL, pL * pL};
  T den = 0;
  for (int k = 0; k < 6; k++) den += T(kDen[k]) * mono[k];
  for (int c = 0; c < 2; c++) {
    const FictRow r = kFict[0][c];
    T n = T(x) * (r.l[0] * pD + r.l[1] * pG + r.l[2] * pL) + T(y) * (r.m[0] * pD + r.m[1] * pG + r.m[2] * pL);
    for (int k = 0; k < 6; k++) n += T(r.q[k]) * mono[k];
    g[c] = double(T(r.scale) * n / den);
  }
}
"""


@pytest.fixture(scope="module")
def fixed(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixed64")
    src, lib = d / "fixed64.cpp", d / "libfixed64.so"
    src.write_text(SOURCE)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(shutil.which(os.environ.get("NVCC", "nvcc")))))
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", os.path.join(PKG_DIR, "csrc"),
                    "-I", os.path.join(cuda, "include"), str(src), "-o", str(lib)], check=True)
    L = ctypes.CDLL(str(lib))
    D = ctypes.c_double
    L.solve.argtypes = [ctypes.c_int, D, D, D, D, ctypes.POINTER(D)]
    L.exact.argtypes = [D, D, D, D, ctypes.POINTER(D)]
    L.exact.restype = None
    return L


def _extremes(fixed, which):
    """Least and largest staged x^gamma, in units of 2^-58: a solved cell's,
    rounded as gamma_cell does, or the composition of a cell without a solve."""
    r = (ctypes.c_int64 * 6)()
    fixed.ranges(r)
    low, most = r[2 * which], r[2 * which + 1]
    return (low + 2) >> 2, max((most - 1 + 2) >> 2, 2 ** 58 - 2 ** 5)


@pytest.mark.parametrize("which,around,centre", [(0, 4, 4), (0, 6, 6), (1, 4 * 4 + 4, 20)])
def test_neighbour_sums_stay_in_range(fixed, which, around, centre):
    """The weighted sum of any cells in range fits 64 bits, and so does the
    increment D0 S1 + D1 S2 with D below 2^-7, its rounding included."""
    a, b = _extremes(fixed, which)
    D = 2 ** 63 - 2 ** 10  # the largest D 2^70
    for s in (around * b - centre * a, around * a - centre * b):
        assert -2 ** 63 <= s < 2 ** 63
        assert abs(2 * (D * s >> 64)) + 1 + 2 ** 10 < 2 ** 63


def test_face_differences_stay_in_range(fixed):
    """(u_n - u_c) 2^4, units of 2^-62, of the variable mobility's fluxes; each
    flux (two products with sums of two D below 2^-5, in units of 2^-65)."""
    a, b = _extremes(fixed, 2)
    u = (b - a) << 4
    assert u < 2 ** 63
    assert 2 * ((2 ** 63 - 2) * u >> 64) + 2 < 2 ** 63


def test_face_sum(fixed):
    """The sum of four fluxes, or its refusal where it leaves 64 bits (or one
    of its two differences does): never a wrapped one."""
    I = ctypes.c_int64
    fixed.sum_of_faces.argtypes = [I, I, I, I, ctypes.POINTER(I)]
    top = 2 ** 63 - 1
    values = [0, 1, -1, 2 ** 61, -2 ** 61, 2 ** 62 - 1, 2 ** 62, -2 ** 62, -2 ** 62 - 1, top, -top, -top - 1]
    rng = np.random.default_rng(0)
    cases = [[int(v) for v in rng.choice(len(values), 4)] for _ in range(4000)]
    t = I()
    refused = 0
    for n, s, e, w in ([values[k] for k in c] for c in cases):
        ok = fixed.sum_of_faces(n, s, e, w, ctypes.byref(t))
        if all(-top - 1 <= v <= top for v in (n - s, e - w, n - s + e - w)):
            assert ok and t.value == n - s + e - w
        else:
            assert not ok
            refused += 1
    assert 400 < refused < 3600


def _solve(L, kind, x, y, d, l):
    g, e = (ctypes.c_double * 2)(), (ctypes.c_double * 2)()
    ok = L.solve(kind, x, y, d, l, g)
    L.exact(x, y, d, l, e)
    return ok, np.array(g), np.array(e)


def test_solve_refuses_fractions_that_add_up_to_more_than_one(fixed):
    """Each phase up to exactly 1 (what nucleation paints), both of them too:
    p = 2^63 twice, whose sum is 2^64."""
    for d in (0.6, 0.95, 1.0 - 2.0 ** -53, 1.0):
        for l in (0.6, 0.95, 1.0 - 2.0 ** -53, 1.0):
            assert not _solve(fixed, 3, 0.3, 0.02, d, l)[0], (d, l)


def test_solve_over_the_square_of_phases(fixed):
    """Whatever solve_fixed accepts is x^gamma: within 64 units of 2^-53 (28 in
    20 million random states), where the FP64 forms are off by thousands."""
    phases = [0.0, 1e-7, 1e-3, 0.2, 0.5, 0.8, 0.999, 1.0 - 1e-9, 1.0 - 2.0 ** -53, 1.0]
    comps = [2.0 ** -11, 0.01, 0.0229, 0.1, 0.3, 0.5, 0.9, 1.0 - 2.0 ** -53]
    taken = 0
    for kind, ds, ls in ((1, phases, [0.0]), (2, [0.0], phases), (3, phases, phases)):
        for d in ds:
            for l in ls:
                for x in comps:
                    for y in comps:
                        ok, g, e = _solve(fixed, kind, x, y, d, l)
                        if ok:
                            taken += 1
                            assert np.all(np.abs(g - e) <= 64 * 2.0 ** -53), (kind, x, y, d, l)
    assert taken > 1000
