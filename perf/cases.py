"""The work that users of this framework have it do, as cases to be timed.

A case is a dict of plain values.  Seven kinds, each through the public classes:

  buildup   a Buildup run advanced by one interval of steps
  loop      the reference's own time-step body, method by method, with its
            numpy arrays going in and out (what a ported script does)
  poisson   one Poisson solve on device arrays: charge -> phi and E
  track     electrons loaded into the store and pushed through a fixed field
  wall      wall test, absorbed rows, wall points, Furman emission
  merge     macro-particle management of a loaded store
  scan      a batch of independent runs advanced together

The ranges: grids of 32 to 1024 nodes a side on rectangular, elliptical,
circular and cut-cell chambers, 10^3 to 2^24 macro-electrons, all three Boris
pushes, both Poisson methods and both management rules.
"""
import functools
import math

import numpy as np
import torch

from openecloud_b200.batch import BatchedBuildup
from openecloud_b200.beam import LHCBeamEndless
from openecloud_b200.buildup import Buildup
from openecloud_b200.grid import Grid
from openecloud_b200.magneticField import multipoleExpansionDevice
from openecloud_b200.particleBoundary import AbsorbArbitraryCutCell, AbsorbElliptical, AbsorbRectangular
from openecloud_b200.particleEmitter import FurmanEmitter
from openecloud_b200.particleManagement import globalRandom, localRandom
from openecloud_b200.particles import Particles
from openecloud_b200.poissonSolver import PoissonSolver

QE = 1.602176565e-19
ME = 9.10938291e-31
EPS0 = 8.85418781762e-12

# Grid's boundType of a chamber
RECT, ELLIPSE, CUTCELL = 0, 1, 3


def listed():
    return [
        # the smallest solves: a sanity-size chamber, where launches count
        dict(name="poisson_rect_33x25", kind="poisson", nx=33, ny=25, lx=0.04, ly=0.03, bound=RECT, method="lu"),
        # the direct solve of a mid-size production chamber (half-axes 45 x 18 mm)
        dict(name="poisson_ellipse_512", kind="poisson", nx=512, ny=512, lx=0.09, ly=0.036, bound=ELLIPSE,
             method="lu"),
        # the iterative solve that the largest grid is run with, from a zero start (first step, restart)
        dict(name="poisson_mg_ellipse_1024", kind="poisson", nx=1024, ny=1024, lx=0.09, ly=0.036, bound=ELLIPSE,
             method="mg"),
        # the standard buildup: 128^2 circle, roulette every 50 steps, half an interval a call
        dict(name="buildup_circle_128", kind="buildup", nx=128, ny=128, lx=0.04, ly=0.04, n=10000, target=100000,
             by=0.0, dt=1e-11, beam=1.1e11, sigma=2e-3, sey=1.6, manage="global", every=50, steps=25),
        # the production buildup: 1024^2 ellipse in a dipole, merging every 10 steps, one interval a call
        dict(name="buildup_ellipse_1024", kind="buildup", nx=1024, ny=1024, lx=0.09, ly=0.036, n=2200000,
             target=2000000, by=8.33, dt=5e-12, beam=1.15e11, sigma=1e-3, sey=1.8, manage="local", every=10,
             steps=10),
        # a ported script: every method of the time step, numpy in and out
        dict(name="loop_ellipse_256x128", kind="loop", nx=256, ny=128, lx=0.09, ly=0.036, n=30000, by=0.1),
        # a few test electrons followed through a fixed field: launches only
        dict(name="track_2000_circle_128", kind="track", nx=128, ny=128, lx=0.04, ly=0.04, bound=ELLIPSE, n=2000,
             order="loaded", btype=0, steps=8),
        # the kernel microbench's store: 2^24 cell-sorted electrons, dipole field
        dict(name="track_2e24_rect_512", kind="track", nx=512, ny=512, lx=0.04, ly=0.04, bound=RECT, n=1 << 24,
             order="cell", btype=1, steps=16),
        # a quadrupole and a cut-cell beam screen, electrons in the order a run holds them (not sorted)
        dict(name="track_1e6_cutcell_300x240", kind="track", nx=300, ny=240, lx=0.044, ly=0.036, bound=CUTCELL,
             n=1000003, order="loaded", btype=2, steps=10),
        # a bunch sweeping part of a large cloud into the wall: absorption and secondary emission
        dict(name="wall_2e6_ellipse_512x256", kind="wall", nx=512, ny=256, lx=0.09, ly=0.036, n=2000000,
             sweep=3e-10),
        # one merge event of the production run
        dict(name="merge_2e6_ellipse_1024", kind="merge", nx=1024, ny=1024, lx=0.09, ly=0.036, n=2200000,
             target=2000000, rule="local"),
        # a small parameter scan: independent runs on uneven grids
        dict(name="scan_6_runs", kind="scan", sizes="96,128,192", runs=6, n=10000, steps=25),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _chamber(rng):
    return rng.choice([(0.04, 0.04), (0.09, 0.036), (0.06, 0.05)])


def draw(rng):
    kind = rng.choice(["poisson", "poisson", "poisson", "buildup", "buildup", "loop", "track", "track", "wall",
                       "merge", "scan"])
    lx, ly = _chamber(rng)
    if kind == "poisson":
        method = rng.choice(["lu", "lu", "mg"])
        nx = _log(rng, 32, 1024) if method == "lu" else _log(rng, 256, 1024)
        ny = min(1024, max(24, int(nx * rng.uniform(0.5, 1.1))))
        return dict(kind=kind, nx=nx, ny=ny, lx=lx, ly=ly, bound=rng.choice([RECT, ELLIPSE]), method=method)
    if kind == "buildup":
        nx = _log(rng, 64, 640)
        n = _log(rng, 3000, 1000000)
        manage = rng.choice(["global", "local"])
        return dict(kind=kind, nx=nx, ny=max(48, int(nx * rng.uniform(0.6, 1.0))), lx=lx, ly=ly, n=n,
                    target=int(n * rng.uniform(0.9, 3.0)), by=rng.choice([0.0, 0.5, 8.33]),
                    dt=rng.choice([5e-12, 1e-11]), beam=rng.uniform(0.5e11, 1.5e11), sigma=rng.choice([1e-3, 2e-3]),
                    sey=rng.uniform(1.2, 2.0), manage=manage, every=10 if manage == "local" else 50,
                    steps=rng.choice([10, 25]))
    if kind == "loop":
        nx = _log(rng, 32, 300)
        return dict(kind=kind, nx=nx, ny=max(24, int(nx * rng.uniform(0.5, 1.0))), lx=lx, ly=ly,
                    n=_log(rng, 1000, 100000), by=rng.choice([0.0, 0.1, 0.5]))
    if kind == "track":
        bound = rng.choice([RECT, ELLIPSE, CUTCELL])
        nx = _log(rng, 32, 1024)
        if bound == CUTCELL:
            nx, (lx, ly) = min(nx, 300), (0.044, 0.036)
        return dict(kind=kind, nx=nx, ny=max(24, int(nx * rng.uniform(0.6, 1.0))), lx=lx, ly=ly, bound=bound,
                    n=_log(rng, 1000, 1 << 24), order=rng.choice(["cell", "loaded"]), btype=rng.choice([0, 1, 2]),
                    steps=rng.choice([4, 10, 16]))
    if kind == "wall":
        nx = _log(rng, 64, 1024)
        return dict(kind=kind, nx=nx, ny=max(48, int(nx * rng.uniform(0.5, 1.0))), lx=lx, ly=ly,
                    n=_log(rng, 10000, 2000000), sweep=rng.uniform(1e-11, 3e-10))
    if kind == "merge":
        nx = _log(rng, 64, 1024)
        n = _log(rng, 10000, 2200000)
        target = int(n * rng.uniform(0.8, 1.2))
        # the roulette's choice of whom to drop depends on the order its warps run in, so its outputs
        # cannot be compared; its cloning rule can
        return dict(kind=kind, nx=nx, ny=max(48, int(nx * rng.uniform(0.5, 1.0))), lx=lx, ly=ly, n=n, target=target,
                    rule=rng.choice(["local", "global"]) if target > n else "local")
    return dict(kind="scan", sizes=",".join(str(_log(rng, 64, 200)) for _ in range(2)), runs=rng.randint(2, 6),
                n=_log(rng, 3000, 20000), steps=rng.choice([10, 25]))


# ------------------------------------------------------------- geometry
def _beam_screen(x, y):
    """A circle of 22 mm flattened at +-18 mm, as an LHC beam screen."""
    return 1 if (x * x + y * y < 0.0219 ** 2 and abs(y) < 0.0175) else 0


@functools.lru_cache(maxsize=None)
def _grid(nx, ny, lx, ly, bound):
    return Grid(nx, ny, lx, ly, bound, boundFunc=_beam_screen if bound == CUTCELL else None)


@functools.lru_cache(maxsize=4)
def _solver(nx, ny, lx, ly, bound):
    return PoissonSolver(_grid(nx, ny, lx, ly, bound))


def _mesh(nx, ny, lx, ly):
    """Node coordinates of the extended grid (ny + 2 rows of nx + 2), f64."""
    dx, dy = lx / (nx - 1.0), ly / (ny - 1.0)
    x = torch.linspace(-lx / 2 - dx, lx / 2 + dx, nx + 2, dtype=torch.float64, device="cuda")
    y = torch.linspace(-ly / 2 - dy, ly / 2 + dy, ny + 2, dtype=torch.float64, device="cuda")
    return x, y


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(g, n):
    return torch.rand(n, dtype=torch.float64, device="cuda", generator=g)


def _inside_rows(case, g, n, fill):
    """n electron rows [x, y, vx, vy, vz, w]: uniform in the chamber scaled by
    `fill`, Maxwellian of 5 eV, weights of a cloud that has been managed."""
    lx, ly, bound = case["lx"], case["ly"], case.get("bound", ELLIPSE)
    pd = torch.empty((n, 6), dtype=torch.float64, device="cuda")
    if bound == ELLIPSE:
        r, a = torch.sqrt(_uniform(g, n)) * fill, _uniform(g, n) * (2 * math.pi)
        pd[:, 0], pd[:, 1] = 0.5 * lx * r * torch.cos(a), 0.5 * ly * r * torch.sin(a)
    else:
        # the beam screen's inscribed box for the cut-cell chamber
        fx, fy = (fill, fill) if bound == RECT else (0.55 * fill, 0.9 * fill)
        pd[:, 0], pd[:, 1] = (_uniform(g, n) - 0.5) * lx * fx, (_uniform(g, n) - 0.5) * ly * fy
    sv = math.sqrt(5.0 * QE / ME)
    pd[:, 2:5] = sv * torch.randn((n, 3), dtype=torch.float64, device="cuda", generator=g)
    pd[:, 5] = (0.2 + 1.8 * _uniform(g, n)) * (1e9 / n)
    return pd


def _blob_field(case, g):
    """[Ex | Ey] on the nodes of 16 Gaussian line charges of 1-4 mm."""
    x, y = _mesh(case["nx"], case["ny"], case["lx"], case["ly"])
    u = _uniform(g, 64).cpu().numpy().reshape(16, 4)
    ex = torch.zeros((y.numel(), x.numel()), dtype=torch.float64, device="cuda")
    ey = torch.zeros_like(ex)
    for a, b, c, d in u:
        rx, ry = x[None, :] - (a - 0.5) * 0.6 * case["lx"], y[:, None] - (b - 0.5) * 0.6 * case["ly"]
        s, q = 1e-3 + 3e-3 * c, (2 * d - 1) * 1e-9
        r2 = rx * rx + ry * ry + 1e-30
        f = q / (2 * math.pi * EPS0) * (1 - torch.exp(-r2 / (2 * s * s))) / r2
        ex += f * rx
        ey += f * ry
    return torch.cat([ex.reshape(-1), ey.reshape(-1)])


def _cloud_charge(case, seed):
    """Charge per node: electrons of a ring-shaped cloud with the noise of
    their number, and the proton beam on the axis."""
    g = _gen(seed)
    lx, ly = case["lx"], case["ly"]
    x, y = _mesh(case["nx"], case["ny"], lx, ly)
    r2 = (2 * x[None, :] / lx) ** 2 + (2 * y[:, None] / ly) ** 2
    phase = _uniform(g, 2).cpu().numpy() * 2 * math.pi
    ring = torch.exp(-((torch.sqrt(r2) - 0.6) / 0.25) ** 2) * (1.0 + 0.3 * torch.sin(40 * x[None, :] / lx + phase[0]) *
                                                              torch.cos(30 * y[:, None] / ly + phase[1]))
    noise = 1.0 + 0.2 * torch.randn(r2.shape, dtype=torch.float64, device="cuda", generator=g)
    rho = -1e-13 * ring * noise
    rho += 2e-12 * torch.exp(-(x[None, :] ** 2 + y[:, None] ** 2) / (2 * 2e-3 ** 2))
    rho[r2 >= 0.998] = 0.0
    return rho.reshape(-1).contiguous()


def _record(rows, held):
    """Rows written into a program's own FP32 record of fixed size (zero
    beyond the last row), as it keeps them for output."""
    held.zero_()
    k = min(rows.shape[0], held.shape[0])
    held[:k].copy_(rows[:k])
    return held


def _held(n, dtype=torch.float32):
    return torch.zeros((int(n), 6), dtype=dtype, device="cuda")


_BOUNDARY = {RECT: AbsorbRectangular, ELLIPSE: AbsorbElliptical, CUTCELL: AbsorbArbitraryCutCell}


# -------------------------------------------------------------- prepare
def prepare(case, seed):
    return _PREPARE[case["kind"]](case, int(seed))


def run(state):
    return _RUN[state["case"]["kind"]](state)


def _prepare_poisson(case, seed):
    ps = _solver(case["nx"], case["ny"], case["lx"], case["ly"], case["bound"]).sibling()
    if case["method"] == "mg":
        ps.method, ps.precond, ps.warmStart = "pcg", "mg", "zero"
        ps.prepare()
    return dict(case=case, ps=ps, q=_cloud_charge(case, seed))


def _run_poisson(st):
    e = st["ps"].solveDevice(st["q"])
    return {"phi": st["ps"].getPhiDevice(), "E": e}


def _prepare_buildup(case, seed):
    grid = _grid(case["nx"], case["ny"], case["lx"], case["ly"], ELLIPSE)
    ps = _solver(case["nx"], case["ny"], case["lx"], case["ly"], ELLIPSE).sibling()
    b = Buildup(nx=case["nx"], ny=case["ny"], lx=case["lx"], ly=case["ly"], boundType=ELLIPSE, n_init=case["n"],
                w_init=1e9 / case["n"], dt=case["dt"], beam_particles=case["beam"], radius_sigma=case["sigma"],
                sey_max=case["sey"], type_b_field=1 if case["by"] else 0, b_const=(0.0, case["by"], 0.0),
                target=case["target"], management=case["manage"], management_every=case["every"],
                n_steps_table=20000, seed=1000 + seed, poisson=ps, grid=grid,
                abs_cap=max(200000, 2 * case["target"]))
    return dict(case=case, b=b, held=_held(1.2 * max(case["n"], case["target"])))


def _run_buildup(st):
    b = st["b"]
    b.run(st["case"]["steps"])
    return {"rows": _record(b.P.getParticleDataDevice(), st["held"]), "phi": b.ps.getPhiDevice(),
            "E": b.ps.getEAtGridPointsDevice()}


def _prepare_loop(case, seed):
    grid = _grid(case["nx"], case["ny"], case["lx"], case["ly"], ELLIPSE)
    ps = _solver(case["nx"], case["ny"], case["lx"], case["ly"], ELLIPSE).sibling()
    P = Particles("electrons", "variableWeight")
    P.setBConst([0.0, case["by"], 0.0])
    bd = AbsorbElliptical(grid, P)
    em = FurmanEmitter(bd, P, seyMax=1.6, seed=seed)
    beam = LHCBeamEndless(grid, 1e-11, nParticles=1.1e11, radiusSigma=0.002, bunchLengthSigma=0.25e-9 * 299792458.0)
    P.setParticleData(_inside_rows(case, _gen(seed), case["n"], 0.98).cpu().numpy())
    return dict(case=case, grid=grid, ps=ps, P=P, bd=bd, em=em, beam=beam, t=1.25e-9,
                held=torch.zeros((int(1.2 * case["n"]), 6), dtype=torch.float32))


def _run_loop(st):
    """One time step as a script writes it: charge, field, push, wall, emission."""
    grid, ps, P, bd, em = st["grid"], st["ps"], st["P"], st["bd"], st["em"]
    P.calcGridWeights(grid)
    P.chargeToGrid(grid)
    ps.solve(P.getChargeOnGrid() + st["beam"].getCharge(st["t"]))
    e = ps.getEAtGridPoints()
    P.eFieldToParticles(grid, e)
    P.borisPush(1e-11, 1 if st["case"]["by"] else 0)
    bd.indexInside()
    bd.saveAbsorbed()
    bd.calculateInteractionPoint()
    bd.calculateNormalVectors()
    em.generateSecondaries()
    P.addAndRemoveParticles(em.getEmittedParticles(), P.getIsInside())
    st["t"] += 1e-11
    return {"rows": _record(torch.from_numpy(P.getParticleData()), st["held"]), "E": e,
            "n": P.getMacroParticleCount()}


def _prepare_track(case, seed):
    g = _gen(seed)
    grid = _grid(case["nx"], case["ny"], case["lx"], case["ly"], case["bound"])
    pd = _inside_rows(case, g, case["n"], 0.97)
    if case["order"] == "cell":
        dx, dy = grid.getDx(), grid.getDy()
        cell = torch.floor((pd[:, 0] + grid.getLxExt() / 2) / dx) + \
            torch.floor((pd[:, 1] + grid.getLyExt() / 2) / dy) * grid.getNxExt()
        pd = pd[torch.argsort(cell, stable=True)].contiguous()
    P = Particles("electrons", "variableWeight", capacity=case["n"])
    P.setBConst([0.0, 0.5, 0.0])
    P._bind(grid)
    field = _blob_field(case, g)
    etab = P.fieldTable(grid, field, 2)
    btab = None
    if case["btype"] == 2:
        btab = P.fieldTable(grid, multipoleExpansionDevice(grid, [0.0, 8.0]), 3)
    return dict(case=case, grid=grid, P=P, bd=_BOUNDARY[case["bound"]](grid, P), etab=etab, btab=btab, rows=pd,
                field=field)


def _run_track(st):
    case, P, grid = st["case"], st["P"], st["grid"]
    P.setParticleData(st["rows"])
    for k in range(case["steps"]):
        P.pushGatherDeposit(grid, st["etab"], 1e-11, case["btype"], st["bd"], bCellTable=st["btab"],
                            refreshScale=k == 0)
    n = case["n"]
    out = {k: v[:n] for k, v in P.soa().items()}
    out["absorbed"] = P.absorbedMask()
    out["charge"] = P.getChargeOnGridFixed()[0]
    return out


def _prepare_wall(case, seed):
    grid = _grid(case["nx"], case["ny"], case["lx"], case["ly"], ELLIPSE)
    g = _gen(seed)
    pd = _inside_rows(case, g, case["n"], 0.995)
    pd[:, 2:5] *= math.sqrt(40.0)  # a cloud kicked by a bunch: 200 eV
    P = Particles("electrons", "variableWeight", capacity=case["n"])
    P.setParticleData(pd)
    bd = AbsorbElliptical(grid, P)
    P._bind(grid)
    # one long free step carries the outer part of the cloud through the wall
    etab = P.fieldTable(grid, torch.zeros(2 * grid.getNpExt(), dtype=torch.float64, device="cuda"), 2)
    P.pushGatherDeposit(grid, etab, case["sweep"], 0, bd)
    return dict(case=case, P=P, bd=bd, em=FurmanEmitter(bd, P, seyMax=1.6, seed=seed),
                held=[_held(case["n"] // 4, torch.float64) for _ in range(2)],
                normals=torch.zeros((case["n"] // 4, 2), dtype=torch.float64, device="cuda"))


def _run_wall(st):
    bd, em = st["bd"], st["em"]
    bd.indexInside()
    bd.saveAbsorbed()
    bd.calculateInteractionPoint()
    bd.calculateNormalVectors()
    sec = em.generateSecondaries()
    return {"rows": _record(bd.getAbsorbedParticlesDevice(), st["held"][0]),
            "normals": _record(bd.getNormalVectorsDevice(), st["normals"]),
            "secondaries": _record(sec, st["held"][1]), "n": [bd.getAbsorbedMacroParticleCount(), sec.shape[0]]}


def _prepare_merge(case, seed):
    grid = _grid(case["nx"], case["ny"], case["lx"], case["ly"], ELLIPSE)
    pd = _inside_rows(case, _gen(seed), case["n"], 0.98)
    P = Particles("electrons", "variableWeight", capacity=int(1.25 * max(case["n"], case["target"])))
    P._bind(grid)
    return dict(case=case, grid=grid, P=P, bd=AbsorbElliptical(grid, P), rows=pd,
                held=_held(1.25 * max(case["n"], case["target"])))


def _run_merge(st):
    case, P = st["case"], st["P"]
    P.setParticleData(st["rows"])
    if case["rule"] == "local":
        localRandom(st["grid"], P, st["bd"], case["target"], seed=3, call=1)
    else:
        globalRandom(st["grid"], P, case["target"], seed=3, call=1)
    rows = P.getParticleDataDevice()
    return {"rows": _record(rows, st["held"]), "n": rows.shape[0]}


def _prepare_scan(case, seed):
    sizes = [int(s) for s in case["sizes"].split(",")]
    cfgs = []
    for i in range(case["runs"]):
        lx, ly = ((0.04, 0.04), (0.09, 0.036))[i % 2]
        cfgs.append(dict(nx=sizes[i % len(sizes)], ny=sizes[i % len(sizes)], lx=lx, ly=ly, boundType=ELLIPSE,
                         n_init=case["n"], target=50000, sey_max=1.2 + 0.8 * i / case["runs"],
                         beam_particles=(0.5 + i / case["runs"]) * 1e11, type_b_field=i % 2,
                         b_const=(0.0, 0.5 * (i % 2), 0.0), seed=1000 * (seed + 1) + i, n_steps_table=5000))
    return dict(case=case, b=BatchedBuildup(cfgs, branches=case["runs"], poisson="lu"),
                held=[_held(4 * case["n"]) for _ in range(case["runs"])])


def _run_scan(st):
    b = st["b"]
    b.run(st["case"]["steps"])
    return [{"rows": _record(r.P.getParticleDataDevice(), h), "phi": r.ps.getPhiDevice()}
            for r, h in zip(b.runs, st["held"])]


_PREPARE = {"poisson": _prepare_poisson, "buildup": _prepare_buildup, "loop": _prepare_loop,
            "track": _prepare_track, "wall": _prepare_wall, "merge": _prepare_merge, "scan": _prepare_scan}
_RUN = {"poisson": _run_poisson, "buildup": _run_buildup, "loop": _run_loop, "track": _run_track,
        "wall": _run_wall, "merge": _run_merge, "scan": _run_scan}


# ----------------------------------------------------------------- work
def work(case):
    """Bytes and operations of one pass.  A particle step reads 28 B and
    writes 24 B of FP32 state (cell, offsets, velocities, weight); a solve
    reads 8 B of charge per node and writes phi and two E components; rows
    exchanged with the caller are six f64."""
    kind = case["kind"]
    if kind == "scan":
        sizes = [int(s) for s in case["sizes"].split(",")]
        nodes = sum((sizes[i % len(sizes)] + 2) ** 2 for i in range(case["runs"]))
        return {"bytes": case["steps"] * (52.0 * case["n"] * case["runs"] + 48.0 * nodes),
                "flops": case["steps"] * (120.0 * case["n"] * case["runs"] + 30.0 * nodes)}
    nodes = (case["nx"] + 2) * (case["ny"] + 2)
    if kind == "poisson":
        return {"bytes": 32.0 * nodes, "flops": 30.0 * nodes}
    n = case["n"]
    if kind == "buildup":
        return {"bytes": case["steps"] * (52.0 * n + 48.0 * nodes), "flops": case["steps"] * (120.0 * n + 30.0 * nodes)}
    if kind == "loop":
        return {"bytes": 52.0 * n + 48.0 * nodes + 48.0 * n, "flops": 120.0 * n + 30.0 * nodes}
    if kind == "track":
        return {"bytes": 48.0 * n + case["steps"] * 52.125 * n + 40.0 * nodes, "flops": case["steps"] * 120.0 * n}
    if kind == "wall":
        lost = min(1.0, 2.0 * case["sweep"] * 5e6 / min(case["lx"], case["ly"]))
        return {"bytes": (12.125 + 180.0 * lost) * n, "flops": (20.0 + 4000.0 * lost) * n}
    return {"bytes": 48.0 * n + 28.0 * case["target"], "flops": 100.0 * n}


# ---------------------------------------------------------------- exact
def exact(case, seed):
    """phi of a solve (conjugate gradients in f64 to rounding) and the
    velocities of a track (Boris steps in f64).  The other kinds carry random
    draws or the store's own representation, which has no 64-bit value."""
    if case["kind"] == "poisson":
        return {"phi": _exact_phi(case, seed), "E": None}
    if case["kind"] == "track":
        out = dict.fromkeys(("cell", "ox", "oy", "absorbed", "charge"))
        out.update(_exact_track(case, seed))
        return out
    return None


def _ellipse_edges(case):
    """Lengths of the parts of the grid's edges inside the chamber, [ny, nx]
    per direction on the extended grid (edge i joins node i to the next one)."""
    nx, ny, lx, ly = case["nx"] + 2, case["ny"] + 2, case["lx"], case["ly"]
    dx, dy = lx / (case["nx"] - 1.0), ly / (case["ny"] - 1.0)
    x = np.linspace(-lx / 2 - dx, lx / 2 + dx, nx)
    y = np.linspace(-ly / 2 - dy, ly / 2 + dy, ny)
    if case["bound"] == RECT:
        ins = ((np.abs(x) < lx / 2)[None, :] & (np.abs(y) < ly / 2)[:, None])
        return ins, np.full((ny, nx), dx), np.full((ny, nx), dy), dx, dy
    ins = x[None, :] ** 2 * (4 / lx ** 2) + y[:, None] ** 2 * (4 / ly ** 2) < 1
    hx = 0.5 * lx * np.sqrt(np.maximum(0.0, 1 - y ** 2 * (4 / ly ** 2)))[:, None]
    hy = 0.5 * ly * np.sqrt(np.maximum(0.0, 1 - x ** 2 * (4 / lx ** 2)))[None, :]
    sx = np.clip(np.minimum(hx, x[None, :] + dx) - np.maximum(-hx, x[None, :] + 0 * hx), 0, dx)
    sy = np.clip(np.minimum(hy, y[:, None] + dy) - np.maximum(-hy, y[:, None] + 0 * hy), 0, dy)
    return ins, sx, sy, dx, dy


def _exact_phi(case, seed):
    """A phi = q with A the finite-integration operator: between neighbours
    eps0 * (dual length) / (edge length inside the chamber), phi = 0 on the wall."""
    ins, sx, sy, dx, dy = _ellipse_edges(case)
    with np.errstate(divide="ignore"):
        wx = torch.as_tensor(np.where(sx > 0, EPS0 * dy / sx, 0.0)).cuda()
        wy = torch.as_tensor(np.where(sy > 0, EPS0 * dx / sy, 0.0)).cuda()
    m = torch.as_tensor(ins).cuda().double()
    diag = wx + wy
    diag[:, 1:] += wx[:, :-1]
    diag[1:, :] += wy[:-1, :]
    dinv = m / torch.where(diag > 0, diag, torch.ones_like(diag))
    ax, ay = wx[:, :-1] * m[:, :-1] * m[:, 1:], wy[:-1, :] * m[:-1, :] * m[1:, :]

    def mul(v):
        r = m * diag * v
        r[:, :-1] -= ax * v[:, 1:]
        r[:, 1:] -= ax * v[:, :-1]
        r[:-1, :] -= ay * v[1:, :]
        r[1:, :] -= ay * v[:-1, :]
        return r

    b = _cloud_charge(case, seed).reshape(m.shape) * m
    phi, best = torch.zeros_like(b), None
    for _ in range(3):  # restarts remove the drift of the recurrence
        r = b - mul(phi)
        z = dinv * r
        p, rz = z.clone(), (r * z).sum()
        for k in range(12000):
            q = mul(p)
            a = rz / (p * q).sum()
            phi += a * p
            r -= a * q
            z = dinv * r
            new = (r * z).sum()
            p = z + (new / rz) * p
            rz = new
            if k % 100 == 99 and float(r.norm()) <= 1e-15 * float(b.norm()):
                break
        res = float((b - mul(phi)).norm())
        if best is not None and res >= 0.5 * best:
            break
        best = res
    return phi.reshape(-1)


def _exact_track(case, seed):
    st = _prepare_track(case, seed)
    g, pd = st["grid"], st["rows"].clone()
    nx, npn, dx, dy = g.getNxExt(), g.getNpExt(), g.getDx(), g.getDy()
    qm, dt = -QE / ME, 1e-11
    fields = [st["field"][:npn], st["field"][npn:]]
    if case["btype"] == 2:
        x, y = _mesh(case["nx"], case["ny"], case["lx"], case["ly"])
        one = torch.ones((y.numel(), x.numel()), dtype=torch.float64, device="cuda")
        fields += [(8.0 * y[:, None] * one).reshape(-1), (8.0 * x[None, :] * one).reshape(-1)]
    for _ in range(case["steps"]):
        cx, cy = (pd[:, 0] + g.getLxExt() / 2) / dx, (pd[:, 1] + g.getLyExt() / 2) / dy
        ix = cx.floor().clamp(0, nx - 2)
        iy = cy.floor().clamp(0, g.getNyExt() - 2)
        fx, fy = cx - ix, cy - iy
        c = (ix + iy * nx).long()
        at = [(1 - fx) * (1 - fy) * f[c] + fx * (1 - fy) * f[c + 1] + (1 - fx) * fy * f[c + nx] +
              fx * fy * f[c + nx + 1] for f in fields]
        vx, vy, vz = pd[:, 2], pd[:, 3], pd[:, 4]
        if case["btype"] == 0:
            vx, vy = vx + qm * dt * at[0], vy + qm * dt * at[1]
        else:
            h = 0.5 * qm * dt
            tx, ty = (torch.zeros_like(vx), torch.full_like(vx, 0.5 * h)) if case["btype"] == 1 else \
                (h * at[2], h * at[3])
            vx, vy = vx + h * at[0], vy + h * at[1]
            ux, uy, uz = vx - vz * ty, vy + vz * tx, vz + vx * ty - vy * tx
            f = 2.0 / (1.0 + tx * tx + ty * ty)
            vx, vy, vz = (vx - uz * ty * f + h * at[0], vy + uz * tx * f + h * at[1],
                          vz + (ux * ty - uy * tx) * f)
        pd[:, 2], pd[:, 3], pd[:, 4] = vx, vy, vz
        pd[:, 0] += dt * vx
        pd[:, 1] += dt * vy
    return {"vx": pd[:, 2], "vy": pd[:, 3], "vz": pd[:, 4], "w": pd[:, 5]}
