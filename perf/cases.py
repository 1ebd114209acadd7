"""What this framework is measured on: the jobs its users run, through its public entry points.

A pass is one job, as a driver program runs it: the initial fields go up from
page-locked host memory, the explicit time steps run (with nucleation calls on
the way where the job has them), the output step's summary and free energy are
taken where the job reports them, and the fields come back into page-locked
host memory.  Handles and host buffers are kept from job to job.

Initial fields follow the workloads of this repository (pfa_gb300/ic.py): a
matrix composition with uniform noise, enriched stripes (2D) or a slab (3D),
and seeded delta / laves particles with the tanh profile, zero-flux ghost ring.

``exact`` restates the model (reference: src/discretization.cu:50-1209,
thermo/parabola625.c, thermo/nucleation.c, src/alloy625.cpp:752-919) in plain
FP64 torch / numpy.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "phasefield-precipitate-aging_gb300"))
from pfa_gb300 import lib  # noqa: E402

# The model parameters at dx = 5 nm (diffusion matrix at the mean composition,
# KKS-stable time step): the values a user's program holds.
_DX = 5e-9
_WIDTH = 10e-9
_PARAMS = {"D_Cr": [3.962273482824986e-18, -3.3982957834732076e-17],
           "D_Nb": [3.0564329013875496e-17, 2.3767238268794082e-16],
           "kappa": [1.7727272727272726e-09] * 2, "omega": [171600000.0] * 2,
           "Lmob": [2.500929077475626e-09] * 2, "alpha": 107000000000.0,
           "dx": _DX, "dy": _DX, "dz": _DX}
_DT = {2: 0.000224275, 3: 0.0001495}
_SIGMA, _UNIT_A, _NUC_SEED = 0.13, 0.352e-9, 42


def _params(dim):
    return dict(_PARAMS, dt=_DT[dim])


# ---------------------------------------------------------------------------
# the cases
def _grid2d(name, nx, ny, steps, precision, **kw):
    c = {"kind": "grid2d", "nx": nx, "ny": ny, "steps": steps, "precision": precision,
         "mask": 5, "mobility": "constant", "nucleation": 0, "particles": 4, "stripes": 1,
         "report": False}
    c.update(kw)
    return dict(c, name=name) if name else c


def _grid3d(name, nx, ny, nz, steps, precision, **kw):
    c = {"kind": "grid3d", "nx": nx, "ny": ny, "nz": nz, "steps": steps, "precision": precision,
         "nucleation": 0, "particles": 8, "report": False}
    c.update(kw)
    return dict(c, name=name) if name else c


def _batch(name, grids, lo, hi, steps, layout):
    c = {"kind": "batch", "grids": grids, "lo": lo, "hi": hi, "steps": steps, "layout": layout}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a test-sized grid: launches and calls are what it costs
        _grid2d("fp64_64x48", 64, 48, 100, "fp64", particles=2),
        # the reference's default kind of run: one small FP64 grid, 1000 steps
        # between outputs, an output step with summary and free energy
        _grid2d("fp64_256", 256, 256, 1000, "fp64", report=True),
        # an ordinary FP64 grid, some tens of steps between frames
        _grid2d("fp64_2048", 2048, 2048, 40, "fp64", stripes=8, particles=16),
        # the reference's 9-point mask on a ragged grid
        _grid2d("fp64_nine_1000x733", 1000, 733, 100, "fp64", mask=9, stripes=4, particles=6),
        # composition-dependent mobility, FP64
        _grid2d("fp64_varmob_512", 512, 512, 60, "fp64", mobility="variable", stripes=2),
        # 3D, FP64
        _grid3d("fp64_3d_128", 128, 128, 128, 40, "fp64"),
        # the small FP32 run: 1000 steps with nucleation every 100 and an output step
        _grid2d("fp32_256", 256, 256, 1000, "fp32", nucleation=100, report=True),
        # a served request of the middle size
        _grid2d("fp32_1024", 1024, 1024, 1000, "fp32", nucleation=100, stripes=4, particles=8),
        # the headline grid: 4096 x 4096, 16 stripes, nucleation every 100 steps
        _grid2d("fp32_4096", 4096, 4096, 500, "fp32", nucleation=100, stripes=16, particles=16),
        # composition-dependent mobility in the FP32 form, ragged
        _grid2d("fp32_varmob_1531x1021", 1531, 1021, 200, "fp32", mobility="variable", stripes=4),
        # 3D, FP32 form, with nucleation
        _grid3d("fp32_3d_256", 256, 256, 256, 300, "fp32", nucleation=100, particles=32),
        # many uneven grids stepped together
        _batch("batch_24", 24, 128, 2048, 200, 3),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def even(n):
        return max(2, n - n % 2)

    kind = rng.choice(["2d64", "2d64", "2d32", "2d32", "2d32", "3d64", "3d32", "batch"])
    if kind == "batch":
        return _batch(None, rng.randint(2, 24), rng.choice([64, 128]), rng.choice([512, 1024, 2048]),
                      even(log(40, 200)), rng.randrange(1 << 20))
    if kind[:2] == "3d":
        n = [log(24, 128 if kind == "3d64" else 256) for _ in range(3)]
        cells = n[0] * n[1] * n[2]
        most = 40 * 128 ** 3 if kind == "3d64" else 300 * 256 ** 3
        hi = max(11, min(400, most // cells))
        return _grid3d(None, n[0], n[1], n[2], log(10, hi), "fp" + kind[2:],
                       particles=rng.randint(1, 12), report=rng.random() < 0.25)
    nx, ny = (log(32, 2048), log(32, 2048)) if kind == "2d64" else (log(48, 4096), log(48, 4096))
    mask, mobility = rng.choice([(5, "constant")] * 3 + [(9, "constant"), (5, "variable")])
    cells = nx * ny
    if kind == "2d64":
        most = 12 * 2048 ** 2 if mobility == "variable" else 40 * 2048 ** 2
        precision = "fp64"
    else:
        most = 300 * 4096 ** 2
        precision = rng.choice(["fp32", "fp32", "fp32k"])
    steps = log(10, max(11, min(1000, most // cells)))
    nuc = 0
    if precision != "fp64" and mobility == "constant" and steps >= 50 and rng.random() < 0.5:
        nuc = 50
        steps -= steps % nuc
    return _grid2d(None, nx, ny, steps, precision, mask=mask, mobility=mobility, nucleation=nuc,
                   particles=rng.randint(1, 10), stripes=rng.randint(0, 4),
                   report=rng.random() < 0.25)


def _cells(case):
    if case["kind"] == "batch":
        return sum(n * n for n in _sides(case))
    return case["nx"] * case["ny"] * case.get("nz", 1)


def work(case):
    """Every explicit step reads and writes the state once: 64 bytes per cell
    in FP64 (four fields), 48 (64) in the FP32 forms (four fields and their
    compensations, packed or not); the fields go up and come back once as
    FP64.  Arithmetic of one cell and step: the gamma solve, the Laplacians
    and both updates in their reduced forms."""
    cells, precision = _cells(case), case.get("precision", "fp32")
    state = 48 if precision == "fp32" else 64
    flops = 120 + 120 * (case.get("mobility") == "variable") + 8 * (case["kind"] == "grid3d")
    return {"bytes": float(cells) * (state * case["steps"] + 64), "flops": float(cells) * flops * case["steps"]}


# ---------------------------------------------------------------------------
# inputs
_XE = np.array([[0.52421634830562147, 0.01299272922003303],
                [0.022966218927631978, 0.24984563695705883],
                [0.37392129441013022, 0.25826261799015571]])
_MATRIX_RANGE = ((0.2794, 0.3288), (0.0202, 0.0269))
_ENRICH_RANGE = ((0.2473, 0.2967), (0.1659, 0.1726))


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _p(x):
    return x ** 3 * (6.0 * x ** 2 - 15.0 * x + 10.0)


def _mirror(a):
    """Fill the ghost ring with the adjacent interior values (in place)."""
    for d in range(a.dim()):
        a.select(d, 0).copy_(a.select(d, 1))
        a.select(d, a.shape[d] - 1).copy_(a.select(d, a.shape[d] - 2))
    return a


def _fields(shape, seed, stripes, particles, stripe_width, radius):
    """Four FP64 fields with the ghost ring on the device, interior `shape`
    (ny, nx) or (nz, ny, nx)."""
    dev = _device()
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=dev).manual_seed(seed)
    matrix = [rng.uniform(*r) for r in _MATRIX_RANGE]
    enrich = [rng.uniform(*r) for r in _ENRICH_RANGE]
    comp = []
    for k in range(2):
        u = torch.rand(shape, generator=gen, device=dev, dtype=torch.float64)
        comp.append(matrix[k] + 0.002 * (2.0 * u - 1.0))
    nx = shape[-1]
    for _ in range(stripes):
        lo = int(rng.integers(0, max(1, nx - stripe_width)))
        for k in range(2):
            comp[k][..., lo:lo + stripe_width] += enrich[k] - matrix[k]
    phi = [torch.zeros(shape, device=dev, dtype=torch.float64) for _ in range(2)]
    centres, tries = [], 0
    apart = 2.0 * radius + 3.0 * _WIDTH / _DX
    while len(centres) < particles and tries < 200 * particles:
        tries += 1
        c = rng.uniform(0.0, 1.0, len(shape)) * (np.array(shape) - 1)
        if all(np.sqrt(np.sum((c - o) ** 2)) >= apart for o in centres):
            centres.append(c)
    pad = int(math.ceil(radius + 3.0 * _WIDTH / _DX)) + 1
    for m, c in enumerate(centres):
        box, r2 = [], 0.0
        for d, n in enumerate(shape):
            lo, hi = max(0, int(c[d]) - pad), min(n, int(c[d]) + pad + 1)
            box.append(slice(lo, hi))
            q = torch.arange(lo, hi, device=dev, dtype=torch.float64) - float(c[d])
            r2 = r2 + (q * q).reshape([-1 if e == d else 1 for e in range(len(shape))])
        box, ph = tuple(box), m % 2
        f = 0.5 - 0.5 * torch.tanh(_DX * (torch.sqrt(r2) - radius) / (_WIDTH / 2))
        w = _p(f)
        for k in range(2):
            comp[k][box] = w * float(_XE[1 + ph][k]) + (1.0 - w) * comp[k][box]
        phi[ph][box] = torch.maximum(phi[ph][box], f)
    out = []
    for a in comp + phi:
        h = torch.empty([n + 2 for n in shape], device=dev, dtype=torch.float64)
        h[(slice(1, -1),) * len(shape)] = a
        out.append(_mirror(h))
    return out


def _inputs(case, seed):
    """One list of four device fields per grid of the case."""
    if case["kind"] == "batch":
        return [_fields((n, n), seed * 1000 + k, 1, 4, max(4, min(64, n // 4)), 8.0)
                for k, n in enumerate(_sides(case))]
    if case["kind"] == "grid3d":
        return [_fields((case["nz"], case["ny"], case["nx"]), seed, 1, case["particles"],
                        max(4, case["nx"] // 8), 6.0)]
    return [_fields((case["ny"], case["nx"]), seed, case["stripes"], case["particles"],
                    max(4, min(64, case["nx"] // 4)), 8.0)]


def _sides(case):
    """Sides of a batch's square grids, log-uniform."""
    rng = np.random.default_rng(case["layout"])
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    return [int(round(math.exp(v))) for v in rng.uniform(lo, hi, case["grids"])]


def _host(shape):
    """A page-locked FP64 host array (numpy, backed by the returned tensor)."""
    return torch.empty(tuple(shape), dtype=torch.float64, pin_memory=torch.cuda.is_available())


def _to_host(fields):
    out = []
    for a in fields:
        h = _host(a.shape)
        h.copy_(a)
        out.append(h.numpy())
    return out


def _mask(case):
    return (lib.five_point_mask if case["mask"] == 5 else lib.nine_point_mask)(_DX, _DX)


def prepare(case, seed):
    grids = [_to_host(f) for f in _inputs(case, seed)]
    if case["kind"] == "batch":
        # one page-locked array per field for all the grids, each reading into its part
        sizes = [g[0].size for g in grids]
        flat = [_host((sum(sizes),)).numpy() for _ in range(4)]
        at = np.cumsum([0] + sizes)
        out = [[a[at[k]:at[k + 1]].reshape(g[0].shape) for a in flat] for k, g in enumerate(grids)]
    else:
        out = [[_host(a.shape).numpy() for a in g] for g in grids]
    s = {"case": case, "in": grids, "out": out}
    if case["kind"] == "batch":
        s["flat"] = flat
        params = _params(2)
        need = sum(lib.Batch.footprint(g[0].shape) for g in grids)
        b = s["batch"] = lib.Batch(params, need)
        slots = [b.add(g) for g in grids]
        b.tune()
        for k in slots:
            b.remove(k)
        b.sync()
        return s
    if case["kind"] == "grid3d":
        g = s["grid"] = lib.Grid3D(grids[0], _params(3), precision=case["precision"])
    else:
        g = s["grid"] = lib.Grid2D(grids[0], _params(2), precision=case["precision"],
                                   mask=_mask(case), mobility=case["mobility"])
    if case["nucleation"]:
        g.set_nucleation(seed=_NUC_SEED, interval=case["nucleation"], sigma=(_SIGMA, _SIGMA),
                         unit_a=_UNIT_A)
    return s


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b = state["batch"]
        slots = [b.add(g) for g in state["in"]]
        b.run(case["steps"])
        for k, o in zip(slots, state["out"]):
            b.read_async(k, o)
        b.sync()
        for k in slots:
            b.remove(k)
        return dict(zip(_NAMES, state["flat"]))
    g = state["grid"]
    g.upload(state["in"][0])
    g.run(case["steps"])
    got = {}
    if case["report"]:
        got["summary"] = g.summarize()
        got["energy"] = g.energy()
    g.read(state["out"][0])
    got.update(zip(_NAMES, state["out"][0]))
    return got


_NAMES = ("x_cr", "x_nb", "phi_del", "phi_lav")


# ---------------------------------------------------------------------------
# the model in FP64, restated (thermo/parabola625.c)
_G = ((2267132212.7620249, 15095482346.486225, 7913298631.5869827, 55193083240.685936),
      (21346492990.798885, 16906497386.287418, 388278320.27291465, 3085369132931.8848),
      (8866730284.8069954, 24191004361.532181, 9045531663.945219, 98294310279.883911))
_DEN = (0.001036042775998007, 0.12229015747171917, 0.041785936156220213, 1.0,
        0.73028945399293654, 0.093983883345629876)
# x^phase_comp = scale (X l.p + Y m.p + q.pp) / (den.pp), p = (p_del, p_gam, p_lav)
_FICT = (
    ((1.0, (0.016938286205500769, 1.0, 0.54889980006097594),
      (-0.3468746660495467, 0.0, -0.10246420218061991),
      (0.086819224054883945, 0.036767802923980249, 0.11815012520929236, 0.0,
       -0.27750258277182049, -0.12951476250779617)),
     (-1.0, (0.0021576593653206376, 0.0, 0.054466450838266962),
      (-0.10535187126621841, -1.0, -0.18138965393196074),
      (0.026258691080522339, 0.24849448207756414, 0.06992726713680375, 0.0,
       0.22257870755542869, 0.025258893954068839))),
    ((0.3468746660495467, (0.0029867928603642137, 0.30371739875396442, 0.11224396861282376),
      (0.0, 1.0, 0.15026949298026254),
      (0.0, -0.25028989589710454, -0.038472217853981416, -0.10599737173866837,
       -0.38426983287411109, -0.074556825343604527)),
     (0.24849448207756414, (0.0, 0.0086829266681549659, 0.0010534256500958396),
      (0.0041692787998190662, 0.068163631095090937, 0.011474488301439056),
      (0.0, 0.10567112340275649, 0.038045328588644858, 1.0, 0.71270814650507497,
       0.091137578230976013))),
    ((0.27750258277182055, (0.010275028791049912, 0.65365032685519298, 0.33867750853659306),
      (-0.18783493715380425, 0.36923693162478488, 0.0),
      (0.04808977843373196, 0.054570103782716275, 0.093195074562756067, 1.0,
       0.46671552103819908, 0.0)),
     (-0.54889980006097605, (0.00047690026722310247, -0.099228403494073802, 0.0),
      (-0.070932051941581864, -1.0, -0.1712222947342838),
      (0.017223643043877624, 0.19525744879034301, 0.041259234012827196, -0.40549970601319757,
       -0.046017313089315913, 0.0))),
)
_HCRCR, _HCRNB, _HNBNB = 45342.644255240499, 150954.82346486227, 1103861.6648137188
_KT = 1.5782889043500002e-20


def _fict(X, Y, pd, pg, pl):
    """The three phases' compositions ((Cr, Nb) each)."""
    lin = (pd, pg, pl)
    mono = (pd * pd, pd * pg, pd * pl, pg * pg, pg * pl, pl * pl)

    def dot(c, v):
        s = 0.0
        for a, b in zip(c, v):
            if a:
                s = s + a * b
        return s

    den = dot(_DEN, mono)
    return [[r[0] * (X * dot(r[1], lin) + Y * dot(r[2], lin) + dot(r[3], mono)) / den for r in row]
            for row in _FICT]


def _g(ph, X, Y):
    A, B, C, E = _G[ph]
    u, v = X - float(_XE[ph][0]), Y - float(_XE[ph][1])
    return A * u * u + (B * X - C) * v + E * v * v


def _dmatrix(X, Y, exp):
    xni = 1.0 - X - Y
    eNb = 1.4170990277916469e-20 * exp(-34.982563536715503 * Y * xni + 14.437947842988088 * Y)
    eCr = 3.5027570743586952e-21 * exp(-7.1543718172640256 * X * xni + 3.3541967644499233 * X)
    eNi = 1.8295676400933012e-21 * exp(-8.5221193705645018 * X * xni + 4.0036674816806448 * X -
                                       442.62877981749585 * Y * xni - 0.82164267100913768 * Y)
    s0, s1 = -_HCRCR * X - _HCRNB * Y, -_HCRNB * X - _HNBNB * Y
    return ((-eNb * X * Y * (s0 + _HCRNB) + eCr * X * (1 - X) * (s0 + _HCRCR) - eNi * X * s0 * xni,
             -eNb * X * Y * (s1 + _HNBNB) + eCr * X * (1 - X) * (s1 + _HCRNB) - eNi * X * s1 * xni),
            (-eCr * X * Y * (s0 + _HCRCR) + eNb * Y * (1 - Y) * (s0 + _HCRNB) - eNi * Y * s0 * xni,
             -eCr * X * Y * (s1 + _HCRNB) + eNb * Y * (1 - Y) * (s1 + _HNBNB) - eNi * Y * s1 * xni))


def _shifted(a, d, by):
    """a's interior moved by one cell along dimension d (a has the ghost ring)."""
    ix = [slice(1, -1)] * a.dim()
    ix[d] = slice(1 + by, a.shape[d] - 1 + by)
    return a[tuple(ix)]


def _laplacian(a, nine):
    c = a[(slice(1, -1),) * a.dim()]
    if nine:
        edge = sum(_shifted(a, d, s) - c for d in range(2) for s in (-1, 1))
        corner = sum(a[1 + i:a.shape[0] - 1 + i, 1 + j:a.shape[1] - 1 + j] - c
                     for i in (-1, 1) for j in (-1, 1))
        return (4.0 * edge + corner) / (6.0 * _DX * _DX)
    return sum(_shifted(a, d, s) - c for d in range(a.dim()) for s in (-1, 1)) / (_DX * _DX)


def _ring(c):
    """c with a zero-flux ghost ring."""
    a = torch.empty([n + 2 for n in c.shape], dtype=c.dtype, device=c.device)
    a[(slice(1, -1),) * c.dim()] = c
    return _mirror(a)


def _step(f, dt, nine, varmob):
    """One explicit step of the four interior fields."""
    X, Y, phd, phl = f
    P = _PARAMS
    pd, pl = _p(phd), _p(phl)
    pg = 1.0 - pd - pl
    xg, xd, xl = _fict(X, Y, pd, pg, pl)
    if varmob:
        D = [[_ring(v) for v in row] for row in _dmatrix(X, Y, torch.exp)]
        u = [_ring(v) for v in xg]
        div = [0.0, 0.0]
        core = (slice(1, -1),) * X.dim()
        for d in range(X.dim()):
            for s in (-1, 1):
                for k in range(2):
                    for j in range(2):
                        div[k] = div[k] + (_shifted(D[k][j], d, s) + D[k][j][core]) * (
                            _shifted(u[j], d, s) - u[j][core])
        new = [X + dt * div[0] / (2 * _DX * _DX), Y + dt * div[1] / (2 * _DX * _DX)]
    else:
        lx, ly = _laplacian(_ring(xg[0]), nine), _laplacian(_ring(xg[1]), nine)
        new = [X + dt * (P["D_Cr"][0] * lx + P["D_Cr"][1] * ly),
               Y + dt * (P["D_Nb"][0] * lx + P["D_Nb"][1] * ly)]
    gg = _g(0, *xg)
    mu0 = 2.0 * _G[0][0] * (xg[0] - float(_XE[0][0])) + _G[0][1] * (xg[1] - float(_XE[0][1]))
    mu1 = _G[0][1] * xg[0] - _G[0][2] + 2.0 * _G[0][3] * (xg[1] - float(_XE[0][1]))
    for k, (a, b, xi) in enumerate(((phd, phl, xd), (phl, phd, xl))):
        gp = gg - _g(k + 1, *xi) - mu0 * (xg[0] - xi[0]) - mu1 * (xg[1] - xi[1])
        pp = 30.0 * a * a * (1.0 - a) * (1.0 - a)
        dF = (-pp * gp + 2.0 * P["omega"][k] * a * (a - 1.0) * (2.0 * a - 1.0) +
              2.0 * P["alpha"] * a * b * b - P["kappa"][k] * _laplacian(_ring(a), nine))
        new.append(a - dt * P["Lmob"][k] * dF)
    return new


def _philox(idx, call, seed):
    """Philox4x32-10 words of counters (idx, call) under key seed (numpy)."""
    m = np.uint64(0xFFFFFFFF)
    sh = np.uint64(32)
    idx = idx.astype(np.uint64)
    c = [idx & m, idx >> sh, np.full_like(idx, call & 0xFFFFFFFF), np.full_like(idx, call >> 32)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> sh) ^ c[1] ^ np.uint64(k0), p1 & m, (p0 >> sh) ^ c[3] ^ np.uint64(k1), p0 & m]
    return c


def _u53(hi, lo):
    k = ((hi << np.uint64(32)) | lo) >> np.uint64(11)
    return (k + np.uint64(1)).astype(np.float64) / 9007199254740992.0


def _nucleate(f, interval, dt, call):
    """One nucleation call on the interior fields, in place (nuclei of less
    than a cell, as the spacing handed to the nucleation kernel makes them in
    2D; in 3D an event would need a ball, and none occurs at these sizes)."""
    X, Y, phd, phl = f
    dim = X.dim()
    d = [_DX] * 3
    if dim == 2:  # the reference hands its kernel dx nx and dy ny, ghost ring included
        d[0], d[1] = _DX * (X.shape[1] + 2), _DX * (X.shape[0] + 2)
    dV = d[0] * d[1] * d[2]
    dt_nuc = interval * dt
    vatom = 0.25 * _UNIT_A ** 3
    n_gam = dV / vatom
    dG = _g(0, X, Y)
    D = _dmatrix(X, Y, torch.exp)
    s3 = _SIGMA ** 3
    zeldov = vatom * dG * dG / (8.0 * math.pi * math.sqrt(_KT * s3))
    gstar = 16.0 * math.pi * s3 / (3.0 * dG * dG)
    k1 = [3.0 * gstar * D[k][k] * (X, Y)[k] / (_SIGMA * 0.352e-9 ** 4) * zeldov * n_gam for k in (0, 1)]
    k2 = gstar / _KT
    J = k1[0] * torch.exp(-k2 / (float(_XE[0][0]) - X)) + k1[1] * torch.exp(-k2 / (Y - float(_XE[0][1])))
    P = 1.0 - torch.exp(-dt_nuc * dV * J)
    R = 2.0 * _SIGMA / dG / d[0]
    ok = (P > 0) & (R > 0) & (_p(phd) + _p(phl) < 1e-10)
    at = torch.nonzero(ok)
    if not len(at):
        return
    pos = at.cpu().numpy().astype(np.int64)
    idx = np.zeros(len(pos), dtype=np.int64)
    for k in range(dim):
        idx = idx * (X.shape[k] + 2) + pos[:, k] + 1
    w = _philox(idx, call, _NUC_SEED)
    u = (_u53(w[0], w[1]), _u53(w[2], w[3]))
    p = P[ok].cpu().numpy()
    r = R[ok].cpu().numpy()
    for k in range(len(pos)):
        for ph in (0, 1):
            if p[k] - u[ph][k] > 0:
                if r[k] > 1.0:
                    raise NotImplementedError("a nucleus of more than one cell")
                c = tuple(int(v) for v in pos[k])
                X[c], Y[c] = float(_XE[1 + ph][0]), float(_XE[1 + ph][1])
                f[2 + ph][c] = 1.0


def _report(f):
    X, Y, phd, phl = f
    P = _PARAMS
    pd, pl = _p(phd), _p(phl)
    pg = 1.0 - pd - pl
    xg, xd, xl = _fict(X, Y, pd, pg, pl)
    dV = _DX ** X.dim()
    e = pg * _g(0, *xg) + pd * _g(1, *xd) + pl * _g(2, *xl)
    e = e + 2.0 * P["alpha"] * phd ** 2 * phl ** 2
    for k, a in enumerate((phd, phl)):
        e = e + P["omega"][k] * a * a * (1.0 - a) ** 2
        r = _ring(a)
        for d in range(a.dim()):
            e = e + P["kappa"][k] * ((_shifted(r, d, 1) - _shifted(r, d, -1)) / (2.0 * _DX)) ** 2
    return {"summary": np.array([float(v.mean()) for v in (X, Y, pg, pd, pl)]),
            "energy": float((e * dV).sum())}


def exact(case, seed):
    dim = 3 if case["kind"] == "grid3d" else 2
    dt, got = _DT[dim], []
    for full in _inputs(case, seed):
        f = [a[(slice(1, -1),) * dim].clone() for a in full]
        nuc, call = case.get("nucleation", 0), 0
        for k in range(case["steps"]):
            f = _step(f, dt, case.get("mask", 5) == 9, case.get("mobility") == "variable")
            if nuc and k % nuc == 0:
                _nucleate(f, nuc, dt, call)
                call += 1
        rep = _report(f) if case.get("report") else {}
        got.append(dict(rep, **dict(zip(_NAMES, (_ring(a).cpu().numpy() for a in f)))))
    if case["kind"] != "batch":
        return got[0]
    return {n: np.concatenate([g[n].reshape(-1) for g in got]) for n in _NAMES}
