"""The FP64 step's linear Allen-Cahn form: what it leaves out stays below the
rounding of the phase for the caller's time step, mobilities and wells, not
only for the workloads'."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle as O
from conftest import PKG_DIR
from pfa_gb300 import ic
from test_fixed64_gpu import step_and_oracle
from test_tiers_gpu import around

SOURCE = r"""
#include "pfa_model.cpp"
using namespace pfa;
// p: dt, then per phase L, kappa, omega, then alpha; out: whether the form is
// taken and, per phase, kw, ka and the five P
extern "C" void coef(const double* p, double* out) {
  ModelConst m{};
  m.dt = p[0];
  for (int i = 0; i < 2; i++) {
    m.L[i] = p[1 + 3 * i];
    m.kappa[i] = p[2 + 3 * i];
    m.omega[i] = p[3 + 3 * i];
  }
  m.alpha = p[7];
  const double mask[9] = {0, 1, 0, 1, -4, 1, 0, 1, 0};
  Coef64 c;
  model_coef64(m, mask, &c);
  out[0] = c.linear;
  for (int i = 0; i < 2; i++) {
    out[1 + 7 * i] = c.kw[i];
    out[2 + 7 * i] = c.ka[i];
    for (int j = 0; j < 5; j++) out[3 + 7 * i + j] = c.P[i][j];
  }
}
"""


def reach(a, corners):
    """Largest magnitude a step reads around each cell."""
    m = around(a)
    if corners:
        for s in (-1, 1):
            for t in (-1, 1):
                m = np.maximum(m, np.abs(np.roll(np.roll(a, s, axis=0), t, axis=1)))
    return m


def test_bounds_follow_the_coefficients(pfa, tmp_path):
    src, lib = tmp_path / "coef.cpp", tmp_path / "libcoef.so"
    src.write_text(SOURCE)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(shutil.which(os.environ.get("NVCC", "nvcc")))))
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(PKG_DIR, "csrc"),
                    "-I", os.path.join(cuda, "include"), str(src), "-o", str(lib)], check=True)
    L = ctypes.CDLL(str(lib))
    p = pfa.model_params()

    def coef(dt=1.0, lmob=1.0, omega=1.0, alpha=1.0):
        a = [p["dt"] * dt]
        for i in range(2):
            a += [p["Lmob"][i] * lmob, p["kappa"][i], p["omega"][i] * omega]
        a.append(p["alpha"] * alpha)
        out = np.zeros(15)
        L.coef(np.array(a, dtype=np.float64).ctypes.data_as(ctypes.c_void_p),
               out.ctypes.data_as(ctypes.c_void_p))
        return out[0], out[1:].reshape(2, 7)

    assert coef()[0] and coef(dt=2.0 / 3.0)[0]  # the workloads'
    taken = 0
    for kw in (dict(), dict(alpha=2.0), dict(alpha=2.0 ** 20), dict(alpha=-1e9), dict(lmob=2.0 ** 20, omega=0.0),
               dict(dt=3.0), dict(dt=1e6), dict(omega=1e12), dict(dt=1e-9), dict(alpha=0.0), dict(dt=1e200),
               dict(alpha=1e150, dt=1e20), dict(dt=np.nan), dict(alpha=np.inf)):
        linear, c = coef(**kw)
        if not linear:
            continue
        taken += 1
        for kwell, ka, c1, c2, c11, c12, c22 in c:
            for u1 in np.linspace(-2.6, 2.6, 9):
                for u2 in np.linspace(-2.6, 2.6, 9):
                    P = u1 * (c1 + c11 * u1 + c12 * u2) + u2 * (c2 + c22 * u2)
                    assert 2.0 ** -60 * abs(P + 3 * kwell) <= 2.0 ** -54
            assert abs(ka) * 2.0 ** -54 <= 2.0 ** -54
    assert 4 <= taken <= 8


# one phase below 2^-60, the other below 2^-27, with a coupling 2^20 times the
# workloads' (one step stays finite); a single phase without well and gradient
# whose driving force is 2^20 times theirs; compositions far outside [0, 1]
@pytest.mark.gpu
@pytest.mark.parametrize("case", ["coupling", "force", "compositions"])
@pytest.mark.parametrize("dim", [2, 3])
def test_linear_form(pfa, orc, case, dim):
    shape = (40, 51) if dim == 2 else (6, 20, 31)
    rng = np.random.default_rng(dim)
    tiny = lambda: 2.0 ** rng.uniform(-62, -59.8, shape)
    f = [rng.uniform(0.28, 0.33, shape), rng.uniform(0.02, 0.17, shape), tiny(), tiny()]
    p, q = pfa.model_params(dim=dim), O.model_params(dim=dim)
    change = {}
    if case == "coupling":
        a = 2.0 ** rng.uniform(-28, -26.8, shape)
        swap = rng.random(shape) < 0.5
        f[2], f[3] = np.where(swap, a, f[2]), np.where(swap, f[3], a)
        change = dict(alpha=p["alpha"] * 2.0 ** 20)
    elif case == "force":
        change = dict(Lmob=[v * 2.0 ** 20 for v in p["Lmob"]], omega=[0.0, 0.0], kappa=[0.0, 0.0])
    else:
        f[0] = rng.choice([-1e9, 0.3, 1e9, 1e12], shape)
    full = []
    for a in f:
        h = np.empty([n + 2 for n in shape])
        h[(slice(1, -1),) * dim] = a
        full.append(ic.mirror_halo(h))
    for k, v in change.items():
        p[k] = v
        if isinstance(v, list):
            getattr(q, k)[:] = v
        else:
            setattr(q, k, v)
    g = (pfa.Grid2D if dim == 2 else pfa.Grid3D)(full, p)
    g.run(1)
    got = g.read()
    g.close()
    want = (orc.run2d if dim == 2 else orc.run3d)(full, q, 1)
    core = (slice(1, -1),) * dim
    # the update's few operations in either form; where compositions are large
    # the driving force's 40, on terms that cancel to 1e-2 of themselves
    rel = (64 if case != "compositions" else 4096) * 2.0 ** -53
    for a, b, o in zip(got[2:], want[2:], full[2:]):
        scale = np.maximum(around(o), np.abs(b))
        assert np.all((np.abs(a - b) <= rel * scale)[core])


# phases from 1e-40 to just below 1e-7, dense at the forms' lines, zero in
# patches: no cell has a solve, so a step rounds each result once in either
# form, and its increments (below 1/100 of the values around) a few times more:
# four last halves of the largest value of the neighbourhood cover both sides
@pytest.mark.gpu
@pytest.mark.parametrize("mask", ["iso", "nine", "five", "variable", "3d"])
@pytest.mark.parametrize("large", [False, True])
def test_forms_without_a_solve(pfa, orc, mask, large):
    if mask == "3d":
        shape = (70, 248, 248) if large else (9, 40, 37)
    else:
        shape = (905, 1000) if large else (93, 130)
    rng = np.random.default_rng(17)
    f = [rng.uniform(0.28, 0.33, shape), rng.uniform(0.02, 0.17, shape)]
    for _ in range(2):
        a = 2.0 ** np.where(rng.random(shape) < 0.5, rng.uniform(-133, -23.5, shape),
                            rng.choice([-60.0, -27.0], shape) + rng.uniform(-0.3, 0.3, shape))
        a = np.minimum(a, 0.99e-7)
        patch = tuple(np.arange(n) // 16 for n in shape)
        zero = rng.random([n // 16 + 1 for n in shape]) < 0.4
        a[zero[np.ix_(*patch)]] = 0.0
        f.append(a)
    got, want = step_and_oracle(pfa, orc, mask, f)
    core = (slice(1, -1),) * len(shape)
    for a, b, o in zip(got, want, f):
        h = np.empty([n + 2 for n in shape])
        h[core] = o
        scale = np.maximum(reach(ic.mirror_halo(h), mask == "nine"), np.abs(b))
        assert np.all((np.abs(a - b) <= 4 * 2.0 ** -53 * scale)[core])
