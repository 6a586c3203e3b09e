"""Timed cases: the work a program has this library do, call by call.

A case is a dict of plain values; `prepare` makes what the program holds
before the call (inputs, grids, correlators, assignors, batches, servers),
`run` is one pass through the public entry points and returns its outputs
whole, `work` counts the bytes and operations the pass cannot do without, and
`exact` recomputes the outputs in 64 bits with plain torch.

Kinds of case:
  survey    Correlator.autocorrelate / cross_correlate of device grids
  periodic  PeriodicCorrelator.autocorrelate of a device grid
  assign    MassAssignor on a catalog in device memory, into a cleared grid
  box       a whole periodic measurement from a catalog in host memory
  batch     PeriodicBatch.run over uneven boxes, and every box's tables
  serve     one survey job (assign, combine, correlate NN and RR) through a
            Server with its grids and correlators resident
"""
import math

import numpy as np
import torch

import fftcorr_b200 as fb
from fftcorr_b200 import batch as fbatch
from fftcorr_b200 import serve as fserve
from fftcorr_b200.catalog.device import DeviceCatalog

NGP, TSC, CIC = 0, 1, 3
NO_WINDOW, TSC_ALIASED = 0, 2

# The survey footprint of the benchmark: a shell sector seen from the origin.
R1, R2, HALF_ANGLE = 500.0, 1500.0, math.radians(30.0)


# ------------------------------------------------------------------- cases

def listed():
    return [
        # A quick look at a small survey on a coarse grid: launch latency.
        dict(name="survey_64_f32_l4", kind="survey", shape="64,64,64", precision="fp32",
             maxell=4, rmax=200.0, dr=10.0, kmax=0.1, dk=0.01, window=TSC_ALIASED,
             cross=False),
        # A periodic box of a simulation suite, start to finish: 100k
        # particles from host memory, CIC, monopole only.
        dict(name="box_128_f64_l0", kind="box", shape="128,128,128", precision="fp64",
             scheme=CIC, n=100_000, boxsize=1000.0, maxell=0, rmax=200.0, dr=10.0,
             kmax=0.2, dk=0.01, window=NO_WINDOW),
        # The plain double-precision survey measurement at a medium grid.
        dict(name="survey_256_f64_l4", kind="survey", shape="256,256,256",
             precision="fp64", maxell=4, rmax=200.0, dr=5.0, kmax=0.2, dk=0.005,
             window=TSC_ALIASED, cross=False),
        # The headline measurement: 512^3, FP32-mixed, ell <= 4.
        dict(name="survey_512_f32_l4", kind="survey", shape="512,512,512",
             precision="fp32", maxell=4, rmax=200.0, dr=5.0, kmax=0.3, dk=0.005,
             window=TSC_ALIASED, cross=False),
        # A wide survey on a fine grid, quadrupole: the largest call.
        dict(name="survey_1024_f32_l2", kind="survey", shape="512,1024,1024",
             precision="fp32", maxell=2, rmax=200.0, dr=5.0, kmax=0.3, dk=0.005,
             window=TSC_ALIASED, cross=False),
        # Two tracers on a grid fitted to the survey, its sides no powers of 2.
        dict(name="survey_cross_ragged_f32_l4", kind="survey", shape="250,360,378",
             precision="fp32", maxell=4, rmax=150.0, dr=5.0, kmax=0.2, dk=0.01,
             window=NO_WINDOW, cross=True),
        # A periodic box of the batched form's largest grid, by itself.
        dict(name="periodic_384_f32_l2", kind="periodic", shape="384,384,384",
             precision="fp32", maxell=2, boxsize=1500.0, rmax=200.0, dr=5.0, kmax=0.1,
             dk=0.005, window=NO_WINDOW),
        # A periodic grid with odd sides in double precision, every multipole.
        dict(name="periodic_odd_f64_l4", kind="periodic", shape="250,243,225",
             precision="fp64", maxell=4, boxsize=1000.0, rmax=150.0, dr=5.0, kmax=0.3,
             dk=0.01, window=TSC_ALIASED),
        # The randoms of the headline job: 100M uniform points of the sector.
        dict(name="assign_tsc_randoms_100M_512_f32", kind="assign", shape="512,512,512",
             precision="fp32", scheme=TSC, n=100_000_000, catalog="sector"),
        # A clustered simulation box of the batched form, FP64 grid.
        dict(name="assign_cic_clustered_8M_384_f64", kind="assign", shape="384,384,384",
             precision="fp64", scheme=CIC, n=8_000_000, catalog="clustered"),
        # Mock boxes of uneven grids and catalogs in one graph.
        dict(name="batch_12_f32_l2", kind="batch", grids="128,192,256,384", nboxes=12,
             precision="fp32", scheme=CIC, nmin=500_000, nmax=8_000_000, pick=4,
             maxell=2, rmax=200.0, dr=5.0, kmax=0.1, dk=0.005, window=NO_WINDOW),
        # A served survey job: 2M clustered galaxies and 20M randoms, xi and P.
        dict(name="serve_survey_256_f32_l4", kind="serve", shape="256,256,256",
             precision="fp32", scheme=TSC, ndata=2_000_000, nrandom=20_000_000,
             maxell=4, rmax=200.0, dr=5.0, kmax=0.2, dk=0.005, window=TSC_ALIASED),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _smooth(n):
    """The nearest size at or below n with no prime factor above 7."""
    while True:
        m = n
        for p in (2, 3, 5, 7):
            while m % p == 0:
                m //= p
        if m == 1:
            return n
        n -= 1


def _grid_side(rng, lo, hi, odd):
    """Mostly the sizes that programs pick (powers of two and their small
    multiples), some of any factorisation when `odd`."""
    n = int(_log(rng, lo, hi))
    how = rng.random()
    if how < 0.35:
        return 1 << max(6, int(math.log2(n) + 0.5))
    if odd and how < 0.6:
        return n
    n = _smooth(n)
    return n if n % 2 == 0 or odd else _smooth(n - n % 2) // 2 * 2


def draw(rng):
    """A case of the listed ranges, without a name."""
    kind = rng.choice(["survey", "survey", "survey", "periodic", "periodic", "assign",
                       "assign", "box", "batch", "serve"])
    precision = rng.choice(["fp32", "fp32", "fp64"])
    odd = rng.random() < 0.3
    window = rng.choice([NO_WINDOW, TSC_ALIASED])
    maxell = rng.choice([0, 2, 4])
    if kind in ("survey", "periodic"):
        limit = 2.0e9 if precision == "fp32" else 0.7e9
        terms = {0: 2, 2: 7, 4: 16}[maxell] if kind == "survey" else 4
        hi = min(640.0, (limit / terms) ** (1.0 / 3.0))
        cube = rng.random() < 0.5
        n0 = _grid_side(rng, 64, hi, odd)
        shape = [n0, n0, n0] if cube else [n0] + [
            _grid_side(rng, max(64, 0.6 * n0), min(1.6 * n0, hi), odd) for _ in range(2)]
        if not odd:
            shape[2] += shape[2] % 2
        while shape[0] * shape[1] * shape[2] * terms > limit:
            shape = [max(64, s // 2) for s in shape]
        case = dict(kind=kind, shape=",".join(map(str, shape)), precision=precision,
                    maxell=maxell, rmax=float(rng.choice([100, 150, 200])),
                    dr=float(rng.choice([2, 5, 10])),
                    kmax=rng.choice([0.1, 0.2, 0.3]), dk=rng.choice([0.005, 0.01]),
                    window=window)
        if kind == "survey":
            case["cross"] = rng.random() < 0.3
        else:
            case["boxsize"] = float(int(rng.uniform(1000, 2000)))
        return case
    if kind == "assign":
        n = int(_log(rng, 1e5, 5e7))
        s = _grid_side(rng, 64, 512, odd)
        return dict(kind=kind, shape=f"{s},{s},{s}", precision=precision,
                    scheme=rng.choice([NGP, TSC, TSC, CIC, CIC]), n=n,
                    catalog=rng.choice(["sector", "clustered"]))
    if kind == "box":
        s = _grid_side(rng, 64, 256, odd)
        return dict(kind=kind, shape=f"{s},{s},{s}", precision=precision,
                    scheme=rng.choice([TSC, CIC]), n=int(_log(rng, 5e4, 1e6)),
                    boxsize=float(int(rng.uniform(1000, 2000))), maxell=maxell,
                    rmax=150.0, dr=10.0, kmax=0.2, dk=0.01, window=window)
    if kind == "batch":
        return dict(kind=kind, grids="128,192,256,384", nboxes=rng.randint(4, 12),
                    precision=precision, scheme=rng.choice([TSC, CIC]), nmin=500_000,
                    nmax=4_000_000, pick=rng.randint(0, 1000), maxell=rng.choice([0, 2]),
                    rmax=200.0, dr=5.0, kmax=0.1, dk=0.005, window=window)
    s = _grid_side(rng, 96, 320, False)
    nd = int(_log(rng, 1e5, 2e6))
    return dict(kind=kind, shape=f"{s},{s},{s}", precision=precision, scheme=TSC,
                ndata=nd, nrandom=nd * rng.randint(3, 10), maxell=maxell, rmax=150.0,
                dr=5.0, kmax=0.2, dk=0.005, window=window)


# ------------------------------------------------------------------ inputs

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)
    return g


def _shape(case):
    return tuple(int(s) for s in case["shape"].split(","))


def _survey_box(shape, sep):
    """posmin and cell size fitting the sector's bounding box, padded as the
    command line does."""
    c = math.cos(HALF_ANGLE)
    y = R2 * math.sin(HALF_ANGLE)
    lo = np.array([R1 * c * c, -y, -y]) - sep / 1.5
    hi = np.array([R2, y, y]) + sep / 1.5
    return lo, max((hi[i] - lo[i]) / shape[i] for i in range(3))


def _in_sector(x, y, z):
    """Whether points lie in the sector (broadcasting coordinates)."""
    rxy2 = x * x + y * y
    r2 = rxy2 + z * z
    t = math.tan(HALF_ANGLE)
    return ((r2 >= R1 * R1) & (r2 < R2 * R2) & (x > 0) & (y.abs() <= t * x) &
            (z * z <= (math.sin(HALF_ANGLE) ** 2) * r2))


def _sector_points(n, gen):
    """n points uniform in the sector, weights U[0.5, 1.5], as (n, 4)."""
    out = torch.empty((n, 4), dtype=torch.float64, device="cuda")
    for s in range(0, n, 1 << 24):
        o = out[s:s + (1 << 24)]
        u = torch.rand((o.shape[0], 4), dtype=torch.float64, device="cuda", generator=gen)
        r = (u[:, 0] * (R2 ** 3 - R1 ** 3) + R1 ** 3) ** (1.0 / 3.0)
        ra = (2 * u[:, 1] - 1) * HALF_ANGLE
        sd = (2 * u[:, 2] - 1) * math.sin(HALF_ANGLE)
        cd = torch.sqrt(1 - sd * sd)
        o[:, 0] = r * cd * torch.cos(ra)
        o[:, 1] = r * cd * torch.sin(ra)
        o[:, 2] = r * sd
        o[:, 3] = 0.5 + u[:, 3]
    return out


def _sector_galaxies(n, gen, ncentres=10000, sigma=5.0):
    """Clumps of width sigma about centres uniform in the sector."""
    c = _sector_points(ncentres, gen)[:, :3]
    out = torch.empty((n, 4), dtype=torch.float64, device="cuda")
    pick = torch.randint(ncentres, (n,), device="cuda", generator=gen)
    out[:, :3] = c[pick] + sigma * torch.randn((n, 3), dtype=torch.float64, device="cuda",
                                               generator=gen)
    out[:, 3] = 0.5 + torch.rand(n, dtype=torch.float64, device="cuda", generator=gen)
    return out


def _box_points(n, boxsize, gen, ncentres=10000, sigma=5.0):
    """A simulation box: half clumps (wrapped), half uniform, unit weights."""
    out = torch.rand((n, 4), dtype=torch.float64, device="cuda", generator=gen)
    out[:, :3] *= boxsize
    h = n // 2
    c = torch.rand((ncentres, 3), dtype=torch.float64, device="cuda", generator=gen) * boxsize
    pick = torch.randint(ncentres, (h,), device="cuda", generator=gen)
    out[:h, :3] = torch.remainder(
        c[pick] + sigma * torch.randn((h, 3), dtype=torch.float64, device="cuda",
                                      generator=gen), boxsize)
    # remainder can round up to the box size itself, which is outside it
    out[:h, :3].clamp_(max=boxsize * (1 - 2.0 ** -52))
    out[:, 3] = 1.0
    # the order of a simulation output: no relation between neighbours in it
    return out[torch.randperm(n, device="cuda", generator=gen)].contiguous()


def _density(case, seed, which=0):
    """A clustered density on the case's grid, in the grid's cell type: a
    smooth random field with shot noise, and for a survey the sector's mask
    (data minus randoms: zero outside it)."""
    shape = _shape(case)
    gen = _gen(2 * seed + which)
    d = torch.randn(shape, dtype=torch.float32, device="cuda", generator=gen)
    f = torch.fft.rfftn(d)
    for a, n in enumerate(shape):
        k = (torch.fft.rfftfreq if a == 2 else torch.fft.fftfreq)(n, device="cuda") * n
        w = 1.0 / (1.0 + (k / 24.0) ** 2)
        f *= w.reshape([-1 if i == a else 1 for i in range(3)])
    s = torch.fft.irfftn(f, s=shape)
    del f
    d = 0.3 * d + s / s.std()
    del s
    if case["kind"] == "survey":
        posmin, cell = _survey_box(shape, case["rmax"])
        ax = [(torch.arange(n, dtype=torch.float32, device="cuda") + 0.5) * cell + float(p)
              for n, p in zip(shape, posmin)]
        for i in range(shape[0]):
            d[i] *= _in_sector(ax[0][i], ax[1][:, None], ax[2][None, :])
    return d if case["precision"] == "fp32" else d.double()


class _Cells:
    """Device memory of the library as an array, which keeps its owner."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape,
                                         "typestr": typestr, "version": 3}


def _cells(grid):
    return torch.as_tensor(_Cells(grid, grid.device_ptr(), grid.shape,
                                  "<f4" if grid.precision == "fp32" else "<f8"),
                           device="cuda")


def _catalog(points):
    """The points as the library's device catalog."""
    cat = DeviceCatalog(points.shape[0])
    torch.as_tensor(_Cells(cat, cat.ptr, tuple(points.shape), "<f8"), device="cuda").copy_(points)
    torch.cuda.synchronize()
    return cat


def _filled_grid(case, cell, posmin, values):
    grid = fb.ConfigSpaceGrid.from_geometry(_shape(case), posmin, cell,
                                            precision=case["precision"])
    _cells(grid).copy_(values)
    torch.cuda.synchronize()
    return grid


def _catalog_points(case, seed):
    gen = _gen(seed)
    if case["catalog"] == "sector":
        return _sector_points(case["n"], gen)
    return _box_points(case["n"], 1000.0, gen)


def _assign_box(case):
    if case["catalog"] == "sector":
        return _survey_box(_shape(case), 200.0)
    return np.zeros(3), 1000.0 / _shape(case)[0]


def _batch_boxes(case):
    """(side, particles, box size) of every box, from the case alone."""
    rng = np.random.default_rng(case["pick"])
    sides = [int(s) for s in case["grids"].split(",")]
    out = []
    for i in range(case["nboxes"]):
        n = math.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"])))
        out.append((sides[i % len(sides)], int(n), float(int(rng.uniform(1000, 2000)))))
    return out


def _serve_points(case, seed):
    gen = _gen(seed)
    return _sector_galaxies(case["ndata"], gen), _sector_points(case["nrandom"], gen)


def _correlator_args(case):
    return dict(rmax=case["rmax"], dr=case["dr"], kmax=case["kmax"], dk=case["dk"],
                maxell=case["maxell"], precision=case["precision"])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "survey":
        shape = _shape(case)
        posmin, cell = _survey_box(shape, case["rmax"])
        corr = fb.Correlator(shape, cell, posmin, case["window"], **_correlator_args(case))
        grid = _filled_grid(case, cell, posmin, _density(case, seed))
        grid2 = _filled_grid(case, cell, posmin, _density(case, seed, 1)) \
            if case["cross"] else None
        return dict(kind=kind, corr=corr, grid=grid, grid2=grid2)
    if kind == "periodic":
        shape = _shape(case)
        cell = case["boxsize"] / max(shape)
        corr = fb.PeriodicCorrelator(shape, cell, case["window"], **_correlator_args(case))
        return dict(kind=kind, corr=corr,
                    grid=_filled_grid(case, cell, np.zeros(3), _density(case, seed)))
    if kind == "assign":
        posmin, cell = _assign_box(case)
        grid = fb.ConfigSpaceGrid.from_geometry(_shape(case), posmin, cell,
                                                precision=case["precision"])
        ma = fb.MassAssignor(grid, fb.DistributionScheme(case["scheme"]),
                             case["catalog"] == "clustered", 0)
        points = _catalog_points(case, seed)
        torch.cuda.synchronize()
        return dict(kind=kind, grid=grid, ma=ma, points=points, cells=_cells(grid))
    if kind == "box":
        shape = _shape(case)
        cell = case["boxsize"] / max(shape)
        grid = fb.ConfigSpaceGrid.from_geometry(shape, np.zeros(3), cell,
                                                precision=case["precision"])
        ma = fb.MassAssignor(grid, fb.DistributionScheme(case["scheme"]), True, 0)
        corr = fb.PeriodicCorrelator(shape, cell, case["window"], **_correlator_args(case))
        points = _box_points(case["n"], case["boxsize"], _gen(seed)).cpu().numpy()
        return dict(kind=kind, grid=grid, ma=ma, corr=corr, points=points,
                    cells=_cells(grid), ncells=float(np.prod(shape)))
    if kind == "batch":
        gen = _gen(seed)
        boxes = [((s, s, s), L / s, _catalog(_box_points(n, L, gen)))
                 for s, n, L in _batch_boxes(case)]
        b = fbatch.PeriodicBatch(boxes, fb.DistributionScheme(case["scheme"]),
                                 window_correct=case["window"], lanes=4, tune=False,
                                 **_correlator_args(case))
        return dict(kind=kind, batch=b, boxes=boxes, precision=case["precision"])
    data, randoms = (_catalog(p) for p in _serve_points(case, seed))
    shape = _shape(case)
    posmin, cell = _survey_box(shape, case["rmax"])
    spec = fserve.JobSpec("survey", shape, cell,
                          fserve.catalog_spec(fserve.CAT_DEVICE, posw=data),
                          fserve.catalog_spec(fserve.CAT_DEVICE, posw=randoms),
                          posmin=posmin, scheme=fb.DistributionScheme(case["scheme"]),
                          window=case["window"], want_rr=True, **_correlator_args(case))
    server = fserve.Server(40 << 30, slots=1)
    state = dict(kind=kind, server=server, spec=spec, precision=case["precision"])
    run(state)  # a server's grids and correlators are built by its first job
    return state


# -------------------------------------------------------------------- runs

def _tables(ps, xi, precision):
    """Both tables' sums and counts (the ratio columns are 0/0 in empty bins),
    in the type of the arithmetic: an FP32-mixed measurement is good to single
    precision, whatever its columns are stored in."""
    real = np.float32 if precision == "fp32" else np.float64
    return [np.asarray(xi["histogram"], real), np.asarray(xi["count"]),
            np.asarray(ps["histogram"], real), np.asarray(ps["count"])]


def run(state):
    kind, corr = state["kind"], state.get("corr")
    if kind == "survey":
        if state["grid2"] is not None:
            return _tables(*corr.cross_correlate(state["grid"], state["grid2"]), corr.precision)
        return _tables(*corr.autocorrelate(state["grid"]), corr.precision)
    if kind == "periodic":
        return _tables(*corr.autocorrelate(state["grid"]), corr.precision)
    if kind == "assign":
        state["grid"].clear()
        state["ma"].clear()
        state["ma"].add_particles_device(state["points"].data_ptr(), state["points"].shape[0])
        return state["cells"]
    if kind == "box":
        grid, ma = state["grid"], state["ma"]
        grid.clear()
        ma.clear()
        ma.add_particles(state["points"])
        totw = ma.totw
        mean = totw / state["ncells"]
        grid -= mean
        grid *= 1.0 / mean
        return _tables(*corr.autocorrelate(grid), corr.precision) + [state["cells"], totw]
    if kind == "batch":
        b = state["batch"]
        b.run()
        out = []
        for i in range(len(b)):
            out += _tables(*b.tables(i), state["precision"])
        return out
    server = state["server"]
    ticket = server.submit(state["spec"])
    server.wait(ticket)
    out = (_tables(*server.tables(ticket, 0), state["precision"]) +
           _tables(*server.tables(ticket, 1), state["precision"]))
    server.release(ticket)
    return out


# -------------------------------------------------------------------- work

def _terms(maxell):
    return {0: 1, 2: 6, 4: 15}[maxell]


def _bins(case):
    rows = case["maxell"] // 2 + 1
    return rows * (case["rmax"] // case["dr"] + case["kmax"] // case["dk"]) * 12


def _fft_flops(cells):
    return 2.5 * cells * math.log2(cells)


def _survey_work(shape, case, grids, cross):
    cells = float(np.prod(shape))
    eb = 4 if case["precision"] == "fp32" else 8
    t = _terms(case["maxell"])
    forward = t + 1 if cross else t  # an autocorrelation's monopole is G itself
    # Every transform crosses its two or three axes; on grids beyond the
    # cache each transform has to touch memory, but the call as such has only
    # to read the grids and write the tables.
    return (grids * cells * eb + _bins(case),
            _fft_flops(cells) * (forward + t) + cells * (20.0 * t))


def _periodic_work(shape, case):
    cells = float(np.prod(shape))
    eb = 4 if case["precision"] == "fp32" else 8
    return cells * eb + _bins(case), 2 * _fft_flops(cells) + 6.0 * cells


def _assign_work(shape, case, n):
    cells = float(np.prod(shape))
    eb = 4 if case["precision"] == "fp32" else 8
    taps = {NGP: 1, TSC: 27, CIC: 8}[case["scheme"]]
    return n * 32.0 + cells * eb, n * (2.0 * taps + 30.0)


def work(case):
    kind = case["kind"]
    if kind == "survey":
        b, f = _survey_work(_shape(case), case, 2 if case["cross"] else 1, case["cross"])
    elif kind == "periodic":
        b, f = _periodic_work(_shape(case), case)
    elif kind == "assign":
        b, f = _assign_work(_shape(case), case, case["n"])
    elif kind == "box":
        b0, f0 = _assign_work(_shape(case), case, case["n"])
        b1, f1 = _periodic_work(_shape(case), case)
        b, f = b0 + b1, f0 + f1
    elif kind == "batch":
        b = f = 0.0
        for s, n, _ in _batch_boxes(case):
            b0, f0 = _assign_work((s, s, s), case, n)
            b1, f1 = _periodic_work((s, s, s), case)
            b, f = b + b0 + b1, f + f0 + f1
    else:
        shape = _shape(case)
        b = f = 0.0
        for n in (case["ndata"], case["nrandom"]):
            b0, f0 = _assign_work(shape, case, n)
            b1, f1 = _survey_work(shape, case, 1, False)
            b, f = b + b0 + b1, f + f0 + f1
    return {"bytes": float(b), "flops": float(f)}


# ------------------------------------------------------------------- exact

def _ylm(ell, m, x, y, z):
    """Real spherical harmonic of even ell <= 4 at (x, y, z), broadcasting;
    0 at the origin for ell > 0."""
    if ell == 0:
        return torch.full((1, 1, 1), 1.0 / math.sqrt(4 * math.pi), dtype=torch.float64,
                          device=x.device)
    x2, y2, z2 = x * x, y * y, z * z
    r2 = x2 + y2 + z2 + 1e-20
    n = math.sqrt((2.0 if m else 1.0) / math.pi)
    if ell == 2:
        c, p = {2: (math.sqrt(15 / 32), lambda: x2 - y2),
                1: (math.sqrt(15 / 8), lambda: x * z),
                0: (math.sqrt(5 / 16), lambda: 2 * z2 - x2 - y2),
                -1: (math.sqrt(15 / 8), lambda: y * z),
                -2: (math.sqrt(15 / 8), lambda: x * y)}[m]
        return n * c * p() / r2
    c, p = {4: (3 / 16 * math.sqrt(35 / 2), lambda: x2 * x2 - 6 * x2 * y2 + y2 * y2),
            3: (3 / 8 * math.sqrt(35), lambda: (x2 - 3 * y2) * z * x),
            2: (3 / 8 * math.sqrt(5 / 2), lambda: (6 * z2 - x2 - y2) * (x2 - y2)),
            1: (9 / 8 * math.sqrt(5), lambda: (4 / 3 * z2 - x2 - y2) * x * z),
            0: (3 / 2, lambda: z2 * z2 - 3 * z2 * (x2 + y2) + 3 / 8 * (x2 + y2) ** 2),
            -1: (9 / 8 * math.sqrt(5), lambda: (4 / 3 * z2 - x2 - y2) * y * z),
            -2: (3 / 8 * math.sqrt(5 / 2), lambda: 2 * x * y * (6 * z2 - x2 - y2)),
            -3: (3 / 8 * math.sqrt(35), lambda: (3 * x2 - y2) * y * z),
            -4: (3 / 16 * math.sqrt(35 / 2), lambda: 4 * x * y * (x2 - y2))}[m]
    return n * c * p() / (r2 * r2)


class _Sub:
    """The r- and k-subgrids of a correlator: axes, bins and window."""

    def __init__(self, shape, cell, case):
        self.shape = shape
        dev = "cuda"
        R = math.ceil(case["rmax"] / cell)
        self.R = R
        ra = torch.arange(2 * R + 1, dtype=torch.float64, device=dev) * cell + (-cell * R)
        knyq = math.pi / cell
        ks, kax, win = [], [], []
        for n in shape:
            s = int(2 * math.ceil(case["kmax"] / (2.0 * knyq / n)) + 1)
            s = s if s <= n else 2 * (n // 2) + 1
            ks.append(s)
            k = (torch.arange(s, dtype=torch.float64, device=dev) * (2.0 * knyq / n) +
                 (-(s // 2)) * 2.0 * knyq / n)
            kax.append(k)
            if case["window"] == NO_WINDOW:
                win.append(torch.ones_like(k))
            else:
                q = torch.sin(k * cell / 2.0) ** 2
                win.append(1 - q + 2.0 / 15.0 * q * q)
        self.ks = ks
        self.r = [ra[:, None, None], ra[None, :, None], ra[None, None, :]]
        self.k = [kax[0][:, None, None], kax[1][None, :, None], kax[2][None, None, :]]
        self.inv_w = 1.0 / (win[0][:, None, None] * win[1][None, :, None] *
                            win[2][None, None, :])
        self.nr = int(math.floor(case["rmax"] / case["dr"]))
        self.nk = int(math.floor(case["kmax"] / case["dk"]))
        self.rbin = self._bin(self.r, case["dr"], self.nr)
        self.kbin = self._bin(self.k, case["dk"], self.nk)

    @staticmethod
    def _bin(ax, size, n):
        d = torch.sqrt(ax[0] * ax[0] + ax[1] * ax[1] + ax[2] * ax[2])
        b = torch.floor(d / size)
        return torch.where(b < n, b, torch.full_like(b, n)).long().reshape(-1)

    def hist(self, values, which):
        b, n = (self.rbin, self.nr) if which == "r" else (self.kbin, self.nk)
        return torch.bincount(b, values.reshape(-1), minlength=n + 1)[:n]

    def counts(self, which):
        b, n = (self.rbin, self.nr) if which == "r" else (self.kbin, self.nk)
        return torch.bincount(b, minlength=n + 1)[:n].to(torch.int32)

    def k_values(self, p):
        """Re of the half-complex p at every cell of the k-subgrid."""
        idx = [(torch.arange(s, device=p.device) - s // 2) % n
               for s, n in zip(self.ks[:2], self.shape[:2])]
        neg = [(-i) % n for i, n in zip(idx, self.shape[:2])]
        oz = self.ks[2] // 2
        re = p.real
        pos = re[idx[0]][:, idx[1]][:, :, :oz + 1]
        ref = re[neg[0]][:, neg[1]][:, :, 1:oz + 1].flip(2)
        return torch.cat([ref, pos], 2)

    def r_values(self, p):
        """The unnormalised inverse transform of p on the r-subgrid."""
        f = p
        for a in (0, 1):
            n = self.shape[a]
            i = (torch.arange(-self.R, self.R + 1, device=p.device)) % n
            f = torch.fft.ifft(f, dim=a, norm="forward").index_select(a, i)
        f = torch.fft.irfft(f, n=self.shape[2], dim=2, norm="forward")
        return f[:, :, torch.arange(-self.R, self.R + 1, device=p.device) % self.shape[2]]


def _rows(rows):
    """Histogram rows as the tables lay them out: squeezed, bins first."""
    h = torch.stack(rows)
    return np.transpose(np.squeeze(h.cpu().numpy()))


def _exact_tables(sub, rrows, krows):
    return [_rows(rrows), sub.counts("r").cpu().numpy(), _rows(krows),
            sub.counts("k").cpu().numpy()]


def _exact_periodic(delta, cell, case):
    shape = tuple(delta.shape)
    sub = _Sub(shape, cell, case)
    f = torch.fft.rfftn(delta)
    f = (f.real ** 2 + f.imag ** 2).to(torch.complex128)
    pk, xr = sub.k_values(f), sub.r_values(f)
    del f
    n = float(np.prod(shape))
    rrows, krows = [], []
    for ell in range(0, case["maxell"] + 1, 2):
        c = math.sqrt(4 * math.pi * (2 * ell + 1))
        krows.append(sub.hist((pk * sub.inv_w * _ylm(ell, 0, *sub.k)) *
                              (c * cell ** 3 / n), "k"))
        rrows.append(sub.hist(xr * _ylm(ell, 0, *sub.r) * (c / n / n), "r"))
    return _exact_tables(sub, rrows, krows)


def _exact_survey(rho1, rho2, posmin, cell, case):
    shape = tuple(rho1.shape)
    sub = _Sub(shape, cell, case)
    n = float(np.prod(shape))
    ax = [torch.arange(m, dtype=torch.float64, device="cuda") + (0.5 + float(p) / cell)
          for m, p in zip(shape, posmin)]
    x, y, z = ax[0][:, None, None], ax[1][None, :, None], ax[2][None, None, :]
    g = torch.fft.rfftn(rho2).conj()
    rrows, krows = [], []
    for ell in range(0, case["maxell"] + 1, 2):
        rs = ks = 0.0
        for m in range(-ell, ell + 1):
            w = rho1.clone()
            for i in range(0, shape[0], 32):
                w[i:i + 32] *= _ylm(ell, m, x[i:i + 32], y, z)
            f = torch.fft.rfftn(w)
            del w
            f *= g
            ks = ks + sub.k_values(f) * (sub.inv_w * _ylm(ell, m, *sub.k))
            rs = rs + sub.r_values(f) * _ylm(ell, m, *sub.r)
            del f
        krows.append(sub.hist(ks * (4 * math.pi), "k"))
        rrows.append(sub.hist(rs * (4 * math.pi / n), "r"))
    return _exact_tables(sub, rrows, krows)


def _exact_assign(points, shape, posmin, cell, scheme, out=None, sign=1.0):
    """The points on a grid in 64 bits (every point inside, or periodic)."""
    if out is None:
        out = torch.zeros(shape, dtype=torch.float64, device="cuda")
    flat = out.view(-1)
    lo = torch.tensor(posmin, dtype=torch.float64, device="cuda")
    n = torch.tensor(shape, device="cuda")
    for s in range(0, points.shape[0], 1 << 23):
        p = points[s:s + (1 << 23)]
        x = (p[:, :3] - lo) / cell
        i = torch.floor(x)
        r = x - i
        i = i.long() % n
        w = p[:, 3] * sign
        if scheme == NGP:
            taps = [(0, torch.ones_like(r))]
        elif scheme == CIC:
            taps = [(0, 1 - r), (1, r)]
        else:
            taps = [(-1, 0.5 * (1 - r) * (1 - r)), (0, 0.5 + r - r * r), (1, 0.5 * r * r)]
        for ox, wx in taps:
            jx = (i[:, 0] + ox) % shape[0]
            for oy, wy in taps:
                jxy = jx * shape[1] + (i[:, 1] + oy) % shape[1]
                wxy = w * wx[:, 0] * wy[:, 1]
                for oz, wz in taps:
                    flat.index_add_(0, jxy * shape[2] + (i[:, 2] + oz) % shape[2],
                                    wxy * wz[:, 2])
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "survey":
        posmin, cell = _survey_box(_shape(case), case["rmax"])
        rho = _density(case, seed).double()
        rho2 = _density(case, seed, 1).double() if case["cross"] else rho
        return _exact_survey(rho, rho2, posmin, cell, case)
    if kind == "periodic":
        cell = case["boxsize"] / max(_shape(case))
        return _exact_periodic(_density(case, seed).double(), cell, case)
    if kind == "assign":
        posmin, cell = _assign_box(case)
        return _exact_assign(_catalog_points(case, seed), _shape(case), posmin, cell,
                             case["scheme"])
    if kind == "box":
        shape = _shape(case)
        cell = case["boxsize"] / max(shape)
        points = _box_points(case["n"], case["boxsize"], _gen(seed))
        d = _exact_assign(points, shape, [0.0] * 3, cell, case["scheme"])
        totw = float(points[:, 3].sum())
        mean = totw / float(np.prod(shape))
        d = (d - mean) * (1.0 / mean)
        return _exact_periodic(d, cell, case) + [d, totw]
    if kind == "batch":
        gen = _gen(seed)
        out = []
        for s, n, L in _batch_boxes(case):
            d = _exact_assign(_box_points(n, L, gen), (s, s, s), [0.0] * 3, L / s,
                              case["scheme"])
            mean = n / float(s) ** 3
            out += _exact_periodic((d - mean) * (1.0 / mean), L / s, case)
        return out
    shape = _shape(case)
    posmin, cell = _survey_box(shape, case["rmax"])
    data, randoms = _serve_points(case, seed)
    alpha = float(data[:, 3].sum()) / float(randoms[:, 3].sum())
    nn = _exact_assign(data, shape, posmin, cell, case["scheme"])
    rr = _exact_assign(randoms, shape, posmin, cell, case["scheme"]) * (-alpha)
    nn += rr
    return (_exact_survey(nn, nn, posmin, cell, case) +
            _exact_survey(rr, rr, posmin, cell, case))
