"""The FP64 step's cheaper forms (zero, far-tail and general phases; the
skipped gamma solve) and its tiles, against the oracle."""
import math

import numpy as np
import pytest

import oracle as O
from conftest import field_err
from pfa_gb300 import ic

pytestmark = pytest.mark.gpu


def mixed_fields(shape, seed):
    """Compositions of the matrix with noise; phases log-uniform from 1e-40 to
    0.3 (both sides of every threshold of the forms), zero in patches."""
    rng = np.random.default_rng(seed)
    f = [rng.uniform(0.28, 0.33, shape), rng.uniform(0.02, 0.17, shape)]
    for _ in range(2):
        a = 10.0 ** rng.uniform(-40, -0.5, shape)
        edges = 10.0 ** rng.choice([-18.1, -18.05, -11.45, -11.42, -7.01, -6.99], shape)
        a = np.where(rng.random(shape) < 0.2, edges, a)
        zero = rng.random([max(1, n // 16) + 1 for n in shape]) < 0.4
        for d in range(len(shape)):
            zero = np.repeat(zero, 16, axis=d)
        a[zero[tuple(slice(0, n) for n in shape)]] = 0.0
        f.append(a)
    out = []
    for a in f:
        h = np.empty([n + 2 for n in shape])
        h[(slice(1, -1),) * len(shape)] = a
        out.append(ic.mirror_halo(h))
    return out


def around(a):
    """Largest magnitude in each cell's neighbourhood (itself and its faces)."""
    m = np.abs(a)
    r = m.copy()
    for d in range(a.ndim):
        for s in (-1, 1):
            r = np.maximum(r, np.roll(m, s, axis=d))
    return r


def check_cells(got, want, rel):
    """Every cell within `rel` of the largest value the step reads around it."""
    core = (slice(1, -1),) * got[0].ndim
    for a, b in zip(got, want):
        scale = around(b)
        assert np.all((np.abs(a - b) <= rel * scale)[core])


# tiles of 8 x 8 cells with the fixed-point solve (up to 12288 of them) and the
# FP64 one, 16 x 8 from 8192 with the 9-point mask; partial tiles on both axes
@pytest.mark.parametrize("nx,ny", [(33, 9), (65, 405), (70, 406), (161, 1621), (191, 1622), (650, 905),
                                   (1001, 797)])
@pytest.mark.parametrize("mask", ["iso", "five", "nine"])
def test_forms_2d(pfa, orc, nx, ny, mask):
    f = mixed_fields((ny, nx), nx * ny)
    p = pfa.model_params()
    q = O.model_params()
    dx, dy = p["dx"], p["dx"] * (1.25 if mask == "five" else 1.0)
    m = pfa.nine_point_mask(dx, dy) if mask == "nine" else pfa.five_point_mask(dx, dy)
    g = pfa.Grid2D(f, dict(p, dy=dy), mask=m)
    g.run(1)
    got = g.read()
    g.close()
    q.dy = dy
    want = orc.run2d(f, q.with_mask(m) if mask == "nine" else q, 1)
    # one step: rounding of a few dozen operations on values of one
    # neighbourhood (the solve's cancellation inside delta: 350)
    check_cells(got, want, 350 * 16 * 2.0 ** -53)


# tiles of 8 x 8 and (from 576 of them) 16 x 16 cells
@pytest.mark.parametrize("nx,ny", [(33, 9), (65, 130), (40, 700), (330, 250), (401, 380)])
def test_forms_varmob(pfa, orc, nx, ny):
    f = mixed_fields((ny, nx), nx + ny)
    g = pfa.Grid2D(f, pfa.model_params(), mobility="variable")
    g.run(1)
    got = g.read()
    g.close()
    check_cells(got, orc.run2d_varmob(f, O.model_params(), 1), 350 * 16 * 2.0 ** -53)


# cells that the fixed-point gamma solve takes beside cells it refuses (a phase
# below 0 or above 1, fractions that add up to more than 1, compositions out of
# range, |x^gamma| of 2 and more), in the sizes that take it (2D up to 12288
# tiles of 8 x 8, 3D up to 65536 planes of tiles)
@pytest.mark.parametrize("mask", ["iso", "nine", "five", "variable", "3d"])
def test_solve_out_of_range(pfa, orc, mask):
    shape = (9, 40, 37) if mask == "3d" else (210, 190)
    rng = np.random.default_rng(7)
    kind = rng.integers(0, 7, shape)
    x, y = rng.uniform(0.28, 0.33, shape), rng.uniform(0.02, 0.17, shape)
    d, l = np.zeros(shape), np.zeros(shape)
    near = kind >= 4  # the precipitates' compositions in half of their cells
    x[near & (kind < 6)], y[near & (kind < 6)] = 0.03, 0.247
    d[kind == 1], l[kind == 1] = 1.0, 0.0
    d[kind == 2], l[kind == 2] = 1.0, 0.05
    d[kind == 3] = -1e-3
    d[kind == 4] = 1.0
    d[kind == 5], l[kind == 5] = 0.5, 1e-9
    l[kind == 6] = rng.choice([1.0 + 1e-12, 0.4, 1.0], shape)[kind == 6]
    y[kind == 6] = rng.choice([1e-5, 0.2], shape)[kind == 6]
    f = []
    for a in (x, y, d, l):
        h = np.empty([n + 2 for n in shape])
        h[(slice(1, -1),) * len(shape)] = a
        f.append(ic.mirror_halo(h))
    p = pfa.model_params(dim=len(shape))
    q = O.model_params(dim=len(shape))
    if mask == "3d":
        g, want = pfa.Grid3D(f, p), orc.run3d(f, q, 1)
    elif mask == "variable":
        g, want = pfa.Grid2D(f, p, mobility="variable"), orc.run2d_varmob(f, q, 1)
    else:
        q.dy = p["dx"] * (1.25 if mask == "five" else 1.0)
        m = (pfa.nine_point_mask if mask == "nine" else pfa.five_point_mask)(p["dx"], q.dy)
        g = pfa.Grid2D(f, dict(p, dy=q.dy), mask=m)
        want = orc.run2d(f, q.with_mask(m) if mask == "nine" else q, 1)
    g.run(1)
    got = g.read()
    g.close()
    check_cells(got, want, 350 * 16 * 2.0 ** -53)


# compositions inside and outside the range of the integer mobilities: Nb below
# 2^-11, Cr and Nb adding up to more than 1, both edges, in one grid and mixed
# within a warp
@pytest.mark.parametrize("nx,ny", [(37, 21), (330, 250), (401, 380)])
def test_mobilities_out_of_range(pfa, orc, nx, ny):
    rng = np.random.default_rng(nx)
    kind = rng.integers(0, 5, (ny, nx))
    kind[: ny // 3] = 0
    x = rng.uniform(0.3, 0.6, (ny, nx))
    y = rng.uniform(0.02, 0.12, (ny, nx))
    x[kind == 1] = 0.95
    y[kind == 1] = rng.uniform(0.049, 0.06, (ny, nx))[kind == 1]
    y[kind == 2] = 10.0 ** rng.uniform(-6, -3, (ny, nx))[kind == 2]
    y[kind == 3] = 2.0 ** -11 * (1 - 2.0 ** -53 * rng.integers(-1, 2, (ny, nx)))[kind == 3]
    x[kind == 4], y[kind == 4] = 0.9375, 0.0625
    f = []
    for a in (x, y, np.zeros((ny, nx)), np.zeros((ny, nx))):
        h = np.empty((ny + 2, nx + 2))
        h[1:-1, 1:-1] = a
        f.append(ic.mirror_halo(h))
    g = pfa.Grid2D(f, pfa.model_params(), mobility="variable")
    g.run(1)
    got = g.read()
    g.close()
    # the oracle's exponents reach 50 (their rounding: 2^-47 of D), increments
    # stay below the values around
    check_cells(got, orc.run2d_varmob(f, O.model_params(), 1), 350 * 16 * 2.0 ** -53)


# segments of 1, 2, 3 and 6 planes; partial tiles on every axis
@pytest.mark.parametrize("n", [(31, 15, 3), (20, 14, 60), (64, 40, 131), (199, 93, 61), (95, 61, 700)])
def test_forms_3d(pfa, orc, n):
    f = mixed_fields(n[::-1], sum(n))
    g = pfa.Grid3D(f, pfa.model_params(dim=3))
    g.run(1)
    got = g.read()
    g.close()
    check_cells(got, orc.run3d(f, O.model_params(dim=3), 1), 350 * 16 * 2.0 ** -53)


# rows with and without a remainder of 32 cells, fewer and more pieces of 32
# than the launch has warps (4864); phases of every range of the forms
@pytest.mark.parametrize("nx,ny", [(33, 9), (5, 305), (700, 433)])
def test_report_forms(pfa, orc, nx, ny):
    f = mixed_fields((ny, nx), nx + ny)
    core = (slice(1, -1), slice(1, -1))
    rng = np.random.default_rng(nx)
    for a in f[2:]:  # down to denormals, and values of the skipped forms
        a[core] = np.where(rng.random((ny, nx)) < 0.3, 10.0 ** rng.uniform(-320, -100, (ny, nx)), a[core])
    for a in f[:2]:  # outside the range of the exact sums
        a[core] = np.where(rng.random((ny, nx)) < 0.02, rng.choice([-1e-3, 1e-5, 1.0], (ny, nx)), a[core])
    for a in f:
        ic.mirror_halo(a)
    p = pfa.model_params()
    for precision in ("fp64", "fp32"):
        g = pfa.Grid2D(f, p, precision=precision)
        g.upload(f)
        e, chem, grad = g.energy(maps=True)
        mean = g.summarize()
        v = g.read()
        g.close()
        want = orc.energy2d(v, p["dx"], p["dx"], p["kappa"], p["omega"], p["alpha"], maps=True)
        assert abs(e - want[0]) <= 1e-12 * abs(want[0])
        for a, b in zip((chem, grad), want[1:]):
            assert np.max(np.abs(a - b)[core]) <= 1e-12 * np.max(np.abs(b[core]))
        X, Y, pd, pl = (a[core] for a in v)
        # where both phases are below 1e-7: a few dozen roundings of gamma's
        # paraboloid and the wells
        tail = np.maximum(np.abs(pd), np.abs(pl)) < 1e-7
        A, B, C, E = 2267132212.7620249, 15095482346.486225, 7913298631.5869827, 55193083240.685936
        du, dv = X - 0.52421634830562147, Y - 0.01299272922003303
        scale = p["dx"] ** 2 * (A * du ** 2 + (np.abs(B * X) + C) * np.abs(dv) + E * dv ** 2
                                + p["omega"][0] * (pd ** 2 + pl ** 2))
        assert np.all((np.abs(chem - want[1])[core] <= 32 * 2.0 ** -53 * scale)[tail])
        P = [a ** 3 * (10 - 15 * a + 6 * a * a) for a in (pd, pl)]
        # the additions of a fixed tree and a cell's own dozen roundings
        for got, a in zip(mean, (X, Y, 1 - P[0] - P[1], *P)):
            exact = math.fsum(a.ravel()) / a.size
            assert abs(got - exact) <= 64 * 2.0 ** -53 * max(abs(exact), np.mean(np.abs(a)))


def test_not_a_number_spreads_as_in_the_plain_forms(pfa, orc):
    """A NaN and an infinity in a composition reach the same cells of the same
    fields as in the oracle's expressions, phases zero or not."""
    f = ic.grid2d(70, 40, seed=3, stripe_width=9, n_particles=1, radius=4.0)
    f[0][10, 50] = np.nan
    f[1][30, 60] = np.inf
    want = orc.run2d(f, O.model_params(), 3)
    g = pfa.Grid2D(f, pfa.model_params())
    g.run(3)
    got = g.read()
    g.close()
    core = (slice(1, -1), slice(1, -1))
    for a, b in zip(got, want):
        assert np.array_equal(np.isfinite(a[core]), np.isfinite(b[core]))
    ok = [np.isfinite(b) for b in want]
    err = field_err([np.where(k, a, 0.0) for a, k in zip(got, ok)],
                    [np.where(k, b, 0.0) for b, k in zip(want, ok)])
    assert max(err) <= 1e-12


# compositions a hair from the powers of two, so that half the cells change
# their exponent in the step
@pytest.mark.parametrize("dim", [2, 3])
def test_exponent_changes(pfa, orc, dim):
    shape = (60, 90) if dim == 2 else (20, 24, 40)
    rng = np.random.default_rng(dim)
    f = []
    for k in range(2):
        a = 2.0 ** -rng.integers(1, 8, shape) * (1.0 + rng.uniform(-2e-4, 2e-4, shape))
        f.append(a)
    f += [np.zeros(shape), np.zeros(shape)]
    full = []
    for a in f:
        h = np.empty([n + 2 for n in shape])
        h[(slice(1, -1),) * dim] = a
        full.append(ic.mirror_halo(h))
    p = pfa.model_params(dim=dim)
    g = (pfa.Grid2D if dim == 2 else pfa.Grid3D)(full, p)
    g.run(1)
    got = g.read()
    g.close()
    want = (orc.run2d if dim == 2 else orc.run3d)(full, O.model_params(dim=dim), 1)
    core = (slice(1, -1),) * dim
    for a, b, o in zip(got[:2], want[:2], full[:2]):
        # one rounding of the sum on each side, and the oracle's of its sums
        # (four or six neighbours of up to 1/2, scaled by D < 1/400)
        assert np.all(np.abs(a - b)[core] <= (np.spacing(np.maximum(a, b)) + 2.0 ** -60)[core])
