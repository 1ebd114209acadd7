"""The edges of the FP64 step's fixed-point forms, one step against the oracle."""
import numpy as np
import pytest

import oracle as O
from pfa_gb300 import ic
from test_tiers_gpu import check_cells

pytestmark = pytest.mark.gpu

# one step: rounding of a few dozen operations on values of one neighbourhood
# (the solve's cancellation inside delta: 350)
TOL = 350 * 16 * 2.0 ** -53


def halo(a):
    h = np.empty([n + 2 for n in a.shape])
    h[(slice(1, -1),) * a.ndim] = a
    return ic.mirror_halo(h)


def step_and_oracle(pfa, orc, mask, fields, **params):
    """One FP64 step of interior fields and the oracle's.  mask: iso, nine,
    five (unequal spacings), variable, 3d."""
    f = [halo(a) for a in fields]
    dim = fields[0].ndim
    p = dict(pfa.model_params(dim=dim), **params)
    q = O.model_params(dim=dim)
    for k, v in params.items():
        if isinstance(v, (list, tuple)):
            getattr(q, k)[:] = v
        else:
            setattr(q, k, v)
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
    return got, want


# cells where both phases are exactly 1 (nuclei of both kinds in one cell), or
# within a few last places of it, beside ordinary ones; the second size of a
# mask takes the FP64 solve (2D: more than 12288 tiles; 3D: more than 65536
# planes of tiles)
@pytest.mark.parametrize("mask", ["iso", "nine", "five", "variable", "3d"])
@pytest.mark.parametrize("large", [False, True])
def test_both_phases_one(pfa, orc, mask, large):
    if mask == "3d":
        shape = (70, 248, 248) if large else (9, 40, 37)
    else:
        shape = (905, 1000) if large else (210, 190)
    rng = np.random.default_rng(3)
    x, y = rng.uniform(0.05, 0.33, shape), rng.uniform(0.02, 0.25, shape)
    d, l = np.zeros(shape), np.zeros(shape)
    both = rng.random(shape) < 0.01
    one = np.array([1.0, 1.0, 1.0 - 2.0 ** -53, 1.0 - 2.0 ** -50])
    d[both], l[both] = rng.choice(one, both.sum()), rng.choice(one, both.sum())
    got, want = step_and_oracle(pfa, orc, mask, [x, y, d, l])
    check_cells(got, want, TOL)


def test_step_after_nuclei_of_both_kinds(pfa, orc):
    """A nucleation call whose rates put delta and laves nuclei into the same
    cells (234 of them), then a step."""
    from golden.make_golden import nuc_struct
    comp = (0.2720, 0.1692)
    f = ic.grid2d(96, 96, seed=5, matrix=comp, enrich=comp, noise=0.0, stripes=[], n_particles=0)
    nuc = dict(sigma=(0.04, 0.05), unit_a=0.352e-9, d=(2e-10, 2e-10, 1.0), dt=1e7)
    g = pfa.Grid2D(f, pfa.model_params())
    g.set_nucleation(seed=99, geometry=pfa.NUC_FIXED_GEOMETRY)
    g.swap()
    g.nucleate(sigma=nuc["sigma"], unit_a=nuc["unit_a"], d=nuc["d"], dt_nuc=nuc["dt"])
    g.swap()
    g.run(1)
    got = g.read()
    g.close()
    want, _, _ = orc.nucleation2d(f, nuc_struct(nuc), 99, 0)
    assert np.sum((want[2] == 1.0) & (want[3] == 1.0)) > 100
    check_cells(got, orc.run2d(want, O.model_params(), 1), TOL)


# x^gamma of the two signs side by side: single cells of a delta domain whose
# x_Nb lies 0.0045 to 0.006 above or below that of their neighbours (x^gamma_Cr
# 0.8 and -0.8), single laves cells (-0.9) in a matrix of x_Cr 0.75.  The second
# size of a mask as above.
@pytest.mark.parametrize("mask", ["iso", "nine", "five", "variable", "3d"])
@pytest.mark.parametrize("large", [False, True])
def test_steep_gamma(pfa, orc, mask, large):
    if mask == "3d":
        shape = (70, 248, 248) if large else (9, 40, 37)
    else:
        shape = (905, 1000) if large else (210, 190)
    rng = np.random.default_rng(11)
    i = np.indices(shape)
    single = np.all(i % 3 == 1, axis=0)
    third = i[-1] * 3 // shape[-1]
    x, y = np.full(shape, 0.02297), np.full(shape, 0.24905)
    d, l = np.ones(shape), np.zeros(shape)
    # (up to 0.0052 in half of the rows: |x^gamma| stays below 1 there)
    step = rng.uniform(0.0045, np.where(i[-2] * 2 < shape[-2], 0.0052, 0.006))
    y[(third == 0) & single] += step[(third == 0) & single]
    y[third == 1] = 0.25385
    y[(third == 1) & single] -= step[(third == 1) & single]
    last = third == 2
    x[last], y[last], d[last] = 0.75, 0.02, 0.0
    last &= single
    x[last] = rng.uniform(0.06, 0.12, shape)[last]
    y[last], l[last] = 0.25, 1.0
    got, want = step_and_oracle(pfa, orc, mask, [x, y, d, l])
    check_cells(got, want, TOL)


# faces whose four fluxes add up to more than 1/4 (the integers' range) with
# every diffusivity and x^gamma in the range of the fixed point, and of either
# sign, at twelve times the usual time step (the constant mobilities, unused,
# scaled down so that the mask keeps its fixed-point form)
@pytest.mark.parametrize("nx,ny", [(60, 45), (400, 390)])
def test_large_fluxes(pfa, orc, nx, ny):
    shape = (ny, nx)
    rng = np.random.default_rng(13)
    i = np.indices(shape)
    single = np.all(i % 3 == 1, axis=0)
    flip = (i[0] // 16 + i[1] // 16) % 2 == 1
    laves = (0.4089737663928951, 0.056577406168092814, 0.0, 1.0)
    delta = (0.0093396110639775015, 0.51067932596175425, 0.590024, 0.0)
    f = []
    for k in range(4):
        a = np.where(single != flip, laves[k], delta[k])
        f.append(a * (1.0 - 0.01 * rng.random(shape)) if k < 2 else a)
    p = pfa.model_params()
    small = {k: [0.25 * v for v in p[k]] for k in ("D_Cr", "D_Nb")}
    got, want = step_and_oracle(pfa, orc, "variable", f, dt=12 * p["dt"], **small)
    assert np.max(np.abs(want[1][1:-1, 1:-1] - f[1])) > 0.27
    check_cells(got, want, TOL)
