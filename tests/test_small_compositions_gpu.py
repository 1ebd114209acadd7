"""The FP64 step's rounding of small compositions, against extended precision:
one step of grids without phases, where x^gamma is the composition itself."""
import numpy as np
import pytest

from pfa_gb300 import ic

pytestmark = pytest.mark.gpu

L = np.longdouble  # 64 bits or more


def _step(f, weights, dt, D):
    """X + dt D lap X in extended precision; weights by offset."""
    core = tuple(slice(1, n - 1) for n in f[0].shape)
    lap = []
    for a in f:
        v = np.zeros([n - 2 for n in a.shape], dtype=L)
        for off, w in weights.items():
            v += L(w) * a[tuple(slice(1 + o, n - 1 + o) for o, n in zip(off, a.shape))].astype(L)
        lap.append(v)
    return [f[k][core].astype(L) + L(dt) * (L(D[k][0]) * lap[0] + L(D[k][1]) * lap[1]) for k in range(2)]


# Neighbourhoods of one binade.  The increment is formed in units of 2^-64 (two
# products, each rounded once, their biases taken out: below 1 unit) from
# compositions in units of 2^-58, whose sum, off by 9 units at most (5 and 7
# points; 9 points: 40), meets D below 1/400 (9 points: a sixth of that): below
# 9 x 64 / 400 units; then one rounding.
@pytest.mark.parametrize("exponent", [-11, -10, -9, -8, -7, -6, -3])
@pytest.mark.parametrize("mask", ["iso", "nine", "3d"])
def test_rounding_of_small_compositions(pfa, mask, exponent):
    shape = (20, 40, 50) if mask == "3d" else (160, 250)
    dim = len(shape)
    rng = np.random.default_rng(23)
    f = []
    for _ in range(2):
        h = np.zeros([n + 2 for n in shape])
        h[(slice(1, -1),) * dim] = 2.0 ** rng.uniform(exponent + 0.05, exponent + 0.95, shape)
        f.append(ic.mirror_halo(h))
    f += [np.zeros_like(f[0]), np.zeros_like(f[0])]
    p = pfa.model_params(dim=dim)
    r2 = 1.0 / p["dx"] ** 2
    if mask == "3d":
        w = {(0, 0, 0): -6.0 * r2}
        for d in range(3):
            for s in (-1, 1):
                w[tuple(s if k == d else 0 for k in range(3))] = r2
        g = pfa.Grid3D(f, p)
    else:
        m = (pfa.nine_point_mask if mask == "nine" else pfa.five_point_mask)(p["dx"], p["dx"])
        w = {(j - 1, i - 1): float(np.ravel(m)[3 * j + i]) for j in range(3) for i in range(3)}
        g = pfa.Grid2D(f, p, mask=m)
    g.run(1)
    got = g.read()
    g.close()
    want = _step(f[:2], w, p["dt"], [p["D_Cr"], p["D_Nb"]])
    unit = 2.0 ** (-12 - exponent)  # 2^-64 in last places
    for a, b in zip(got[:2], want):
        a = a[(slice(1, -1),) * dim]
        err = np.abs((a.astype(L) - b) / np.spacing(np.minimum(a, b.astype(np.float64))))
        assert np.max(err) <= 0.5 + unit * (1 + 9 * 64 / 400) + 0.02
        if exponent >= -8:  # as good as FP64's, 0.25
            assert np.mean(err) <= 0.26
