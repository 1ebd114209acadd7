"""Nuclei wider than the grid: the reference bounds-checks the linear cell
index only, so a box wider than a row wraps onto the next rows and meets cells
twice; its serial order decides, here as in the oracle."""
import numpy as np
import pytest

from pfa_gb300 import ic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nx,ny,seed", [(1, 90, 1), (3, 60, 2), (4, 50, 3), (6, 70, 4)])
def test_painting_follows_the_serial_order(pfa, orc, precision, nx, ny, seed):
    from golden.make_golden import nuc_struct
    rng = np.random.default_rng(seed)
    f = []
    for a in (rng.uniform(0.3, 0.5, (ny, nx)), rng.uniform(0.1, 0.25, (ny, nx)), np.zeros((ny, nx)),
              np.zeros((ny, nx))):
        h = np.empty((ny + 2, nx + 2))
        h[1:-1, 1:-1] = a
        f.append(ic.mirror_halo(h))
    d = 3e-11
    nuc = dict(sigma=(0.04, 0.05), unit_a=0.352e-9, d=(d, d, (2e-10 / d) ** 2), dt=1e9)
    p = pfa.model_params()
    g = pfa.Grid2D(f, p, precision=precision)
    g.set_nucleation(seed=seed, geometry=pfa.NUC_FIXED_GEOMETRY)
    if precision == "fp64":
        g.swap()
    g.nucleate(sigma=nuc["sigma"], unit_a=nuc["unit_a"], d=nuc["d"], dt_nuc=nuc["dt"])
    ev = g.events()
    if precision == "fp64":
        g.swap()
    got = g.read()
    g.close()
    want, events, _ = orc.nucleation2d(f, nuc_struct(nuc), seed, 0)
    assert [(e[0], e[1]) for e in events] == ev
    assert sum(2 * e[4] > nx + 2 for e in events) > 5
    core = (slice(1, -1),) * 2
    for a, b in zip(got, want):
        if precision == "fp64":
            assert np.array_equal(a, b)
        else:  # the records' resolution
            assert np.max(np.abs(a - b)[core]) <= 2.0 ** -38
