"""The launcher's row and plane splits: a step's result does not depend on them."""
import numpy as np
import pytest

from pfa_gb300 import ic

pytestmark = pytest.mark.gpu


# sizes on both sides of the split rule's lines (152 SMs: one-row segments up
# to 1368 CTA rows, three-row segments up to 8208, six-row ones above), one
# strip and more, and row counts that leave remainders of the unrolled loop
@pytest.mark.parametrize("nx,ny", [(1, 1), (30, 2), (31, 7), (120, 1368), (121, 685), (481, 275),
                                   (500, 1643), (361, 2741)])
def test_rows_split_is_bit_neutral(pfa, nx, ny):
    """A grid alone (the launcher's split) against the same grid in a batch
    whose units are whole columns: the same bits."""
    f = ic.grid2d(nx, ny, seed=nx + ny, stripe_width=max(1, nx // 4),
                  n_particles=2 if min(nx, ny) > 40 else 0)
    p = pfa.model_params()
    g = pfa.Grid2D(f, p, precision="fp32")
    g.run(5)
    alone = g.read()
    g.close()
    b = pfa.Batch(p, pfa.Batch.footprint(f[0].shape))
    k = b.add(f)
    b.set_launch(1 << 30, True)
    b.run(5)
    whole = b.read(k)
    b.close()
    for x, y in zip(alone, whole):
        assert np.array_equal(x[1:-1, 1:-1], y[1:-1, 1:-1])


@pytest.mark.parametrize("n", [(20, 14, 3), (33, 27, 1), (40, 30, 35), (64, 26, 97)])
def test_plane_split_3d(pfa, n):
    """Short z segments (small 3D grids): the FP32 form against FP64."""
    f = ic.grid3d(*n, seed=sum(n), slab=max(1, n[0] // 4), n_particles=1 if min(n) > 20 else 0)
    p = pfa.model_params(dim=3)
    out = []
    for prec in ("fp64", "fp32"):
        g = pfa.Grid3D(f, p, precision=prec)
        g.run(20)
        out.append(g.read())
        g.close()
    for x, y in zip(*out):
        # the FP32 form's resolution is 2^-40 and its increments of a few
        # 1e-4 per step are rounded to 2^-24 of themselves
        assert np.max(np.abs(x - y)) <= 2e-8
