"""The launcher's row and plane splits: a step's result does not depend on them."""
import numpy as np
import pytest

from pfa_gb300 import ic

pytestmark = pytest.mark.gpu


# sizes on both sides of the split rule's line (152 SMs: one-row segments up
# to 1368 CTA rows, three-row segments above), one strip and more, and row
# counts that leave remainders of the unrolled loop
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


# more segments of the usual height than a launch grid's second dimension holds
@pytest.mark.parametrize("precision,nx,ny", [("fp32", 1, 196609), ("fp32", 2, 400001), ("fp64", 1, 530001)])
def test_tall_grids(pfa, precision, nx, ny):
    """A column without neighbours in x: the same values as in a 64-row piece
    of it, away from the piece's ends."""
    f = ic.grid2d(nx, ny, seed=ny, stripe_width=0, n_particles=0)
    p = pfa.model_params()
    out = []
    for top in (0, ny - 64, ny):
        part = [np.ascontiguousarray(a[top:top + 66]) for a in f] if top < ny else f
        if top < ny:
            for a in part:
                ic.mirror_halo(a)
        g = pfa.Grid2D(part, p, precision=precision)
        for n in (1, 2):
            g.run(n)
        out.append(g.read())
        g.close()
    low, high, whole = out
    for a, b, c in zip(low, high, whole):
        assert np.array_equal(a[1:61, 1:-1], c[1:61, 1:-1])
        assert np.array_equal(b[5:65, 1:-1], c[ny - 59:ny + 1, 1:-1])


@pytest.mark.parametrize("dim", [2, 3])
def test_record_conversions(pfa, dim):
    """Upload and read back without a step: FP32 value and 16-bit count of each
    field, recombined exactly, for every range of the conversions."""
    shape = (90, 71) if dim == 2 else (9, 21, 35)
    rng = np.random.default_rng(dim)
    f, want = [], []
    for k in range(4):
        v = 10.0 ** rng.uniform(-46, 1, shape) * rng.choice([-1.0, 1.0], shape)
        edge = rng.choice([0.0, -0.0, 2.0 ** -29, 2.0 ** -29 * (1 - 2.0 ** -24), 1.0, 2.0, 2.0 * (1 - 2.0 ** -24),
                           2.0 - 2.0 ** -26, 2.0 ** -75, 1e-40, 1e300], shape)
        v = np.where(rng.random(shape) < 0.5, edge, v)
        if k < 2:
            v = np.where(rng.random(shape) < 0.5, rng.uniform(0.01, 0.6, shape), v)
        h = np.empty([n + 2 for n in shape])
        h[(slice(1, -1),) * dim] = v
        f.append(ic.mirror_halo(h))
        with np.errstate(over="ignore", under="ignore", invalid="ignore"):
            hi = f[-1].astype(np.float32)
            c = (hi.astype(np.float64) - f[-1]).astype(np.float32)
            unit = 2.0 ** (40 if k < 2 else 39)
            n = np.clip(np.rint(c.astype(np.float64) * unit), -32768, 32767)
            want.append(hi.astype(np.float64) - n / unit)
    g = (pfa.Grid2D if dim == 2 else pfa.Grid3D)(f, pfa.model_params(dim=dim), precision="fp32")
    g.upload(f)
    if dim == 3:  # (the FP64 fields stay in place until a step or a read of the records converts them)
        raw = np.empty(int(g.L.pfa3d_f32_state_bytes(g.h)), dtype=np.uint8)
        assert g.L.pfa3d_read_f32_state(g.h, raw.ctypes.data, raw.size) == 0
    got = g.read()
    g.close()
    core = (slice(1, -1),) * dim
    for a, b in zip(got, want):
        assert np.array_equal(a[core], b[core])


# segments of four rows (variable mobility, from four CTA rows per resident
# CTA on) with remainders of one to three rows, against a piece in shorter ones
@pytest.mark.parametrize("precision", ["fp32", "fp32k"])
@pytest.mark.parametrize("nx,ny", [(1001, 609), (1001, 610), (1001, 611)])
def test_four_row_segments(pfa, precision, nx, ny):
    f = ic.grid2d(nx, ny, seed=ny, stripe_width=300, n_particles=6)
    out = []
    for top in (ny - 64, ny):
        part = [np.ascontiguousarray(a[top:top + 66]) for a in f] if top < ny else f
        if top < ny:
            for a in part:
                ic.mirror_halo(a)
        g = pfa.Grid2D(part, pfa.model_params(), precision=precision, mobility="variable")
        for _ in range(3):
            g.run(1)
        out.append(g.read())
        g.close()
    for a, b in zip(*out):
        assert np.array_equal(a[5:65, 1:-1], b[ny - 59:ny + 1, 1:-1])


# strips of 28 and 30 columns (double and single passes) put the same cells in
# different warps: tails that cross the bulk threshold of the gamma solve
# everywhere must not notice
def test_strip_width_is_bit_neutral(pfa):
    nx, ny = 1500, 1500
    f = ic.grid2d(nx, ny, seed=4, n_particles=0)
    rng = np.random.default_rng(4)
    for a in f[2:]:
        a[1:-1, 1:-1] = 10.0 ** rng.uniform(-7, -3, (ny, nx))
        ic.mirror_halo(a)
    out = []
    for single in (False, True):
        g = pfa.Grid2D(f, pfa.model_params(), precision="fp32")
        for n in ([1] * 12 if single else [12]):
            g.run(n)
        out.append(g.read())
        g.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y)


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


# launches of several steps on tiles (grids of up to 912 tiles of 26 x 10
# cells): domains inside one tile, partial tiles, edges on every side; 13 steps
# are passes of different lengths
@pytest.mark.parametrize("kind", ["fp32", "fp32k", "nine", "variable"])
@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 35), (18, 2), (61, 5), (64, 48), (129, 131), (257, 255),
                                   (1, 9000), (450, 448)])
def test_tile_steps_are_bit_neutral(pfa, kind, nx, ny):
    f = ic.grid2d(nx, ny, seed=nx + 7 * ny, stripe_width=max(1, nx // 4),
                  n_particles=3 if min(nx, ny) > 40 else 0)
    rng = np.random.default_rng(nx)
    if min(nx, ny) <= 40:  # phases everywhere, some of them zero
        for a in f[2:]:
            a[1:-1, 1:-1] = rng.choice([0.0, 1e-9, 0.2, 0.5], (ny, nx))
            ic.mirror_halo(a)
    kw = {"nine": {"mask": pfa.nine_point_mask(5e-9, 5e-9)}, "variable": {"mobility": "variable"}}.get(kind, {})
    out = []
    for single in (False, True):
        g = pfa.Grid2D(f, pfa.model_params(), precision="fp32k" if kind == "fp32k" else "fp32", **kw)
        for n in ([1] * 13 if single else [13]):
            g.run(n)
        out.append(g.read())
        g.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y)


# record sets just above the line for double steps (96 MB): ragged columns
# (the last strip of 28 one to three columns wide), one-strip and one-row
# grids, row counts that leave remainders
@pytest.mark.parametrize("precision,mask,nx,ny", [
    ("fp32", 5, 1401, 1450), ("fp32", 5, 1430, 1403), ("fp32", 5, 29, 64000), ("fp32", 5, 1, 64001),
    ("fp32", 5, 2000001, 1), ("fp32", 5, 1000002, 2), ("fp32k", 5, 1431, 1100),
    ("fp32", 9, 1402, 1451), ("fp32k", 9, 1429, 1101)])
def test_double_steps_are_bit_neutral(pfa, precision, mask, nx, ny):
    """Runs of double passes (with single steps around the nucleation calls
    and at odd ends) against the same steps one call at a time: the same
    bits, events and counters."""
    small = min(nx, ny) < 60
    f = ic.grid2d(nx, ny, seed=nx + ny, stripe_width=max(1, min(64, nx // 4)),
                  n_particles=0 if small else 6, radius=5.0)
    if small:  # phases along the edges and across the strips
        rng = np.random.default_rng(1)
        for a in f[2:]:
            a[1:-1, 1:-1] = 0.3 * (rng.random((ny, nx)) < 0.1)
            ic.mirror_halo(a)
    p = pfa.model_params()
    m = (pfa.nine_point_mask if mask == 9 else pfa.five_point_mask)(p["dx"], p["dx"])
    out = []
    for single in (False, True):
        g = pfa.Grid2D(f, p, precision=precision, mask=m)
        g.set_nucleation(seed=7, interval=5)
        for n in (11, 4, 7):
            if single:
                for _ in range(n):
                    g.run(1)
            else:
                g.run(n)
        out.append((g.read(), g.events()))
        g.close()
    for x, y in zip(out[0][0], out[1][0]):
        assert np.array_equal(x[1:-1, 1:-1], y[1:-1, 1:-1])
    assert out[0][1] == out[1][1]


@pytest.mark.parametrize("persistent,rows", [(True, 0), (False, 9), (True, 1 << 30)])
def test_batch_double_steps_are_bit_neutral(pfa, persistent, rows):
    """A batch above the line for double passes: runs of even and odd lengths,
    with a member leaving in between, against each grid alone."""
    p = pfa.model_params()
    shapes = [(29, 3), (640, 1200), (1117, 900), (28, 28)]
    fs = [ic.grid2d(nx, ny, seed=k, stripe_width=max(1, nx // 4),
                    n_particles=3 if min(nx, ny) > 60 else 0) for k, (nx, ny) in enumerate(shapes)]
    fs.append(ic.grid2d(500, 700, seed=9))
    b = pfa.Batch(p, sum(pfa.Batch.footprint(f[0].shape) for f in fs))
    slots = [b.add(f) for f in fs]
    if rows:
        b.set_launch(rows, persistent)
    b.run(9)
    b.run(4)
    gone = b.read(slots[4])
    b.remove(slots[4])
    b.run(1)
    b.run(6)
    got = [b.read(k) for k in slots[:4]] + [gone]
    b.close()
    for f, x, n in zip(fs, got, (20, 20, 20, 20, 13)):
        g = pfa.Grid2D(f, p, precision="fp32")
        for _ in range(n):
            g.run(1)
        for u, v in zip(g.read(), x):
            assert np.array_equal(u[1:-1, 1:-1], v[1:-1, 1:-1])
        g.close()
