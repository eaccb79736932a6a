"""The calls whose speed matters to a user of this package, as cases to be timed.

Each case is one pass through a public entry point at a size, layout and precision that real
programs use: the neighbor search alone and behind the reference's own interfaces, a scene's
steps and its solver's right-hand side, a batch of served scenes, and a differentiable
rollout with its gradient.  `exact` restates the results in 64 bits with plain torch.
"""
import math

import numpy as np
import torch

from pytorchsph_gb300 import modules, neighborhoods, workloads
from pytorchsph_gb300.adjoint import DropRollout, drop_rollout
from pytorchsph_gb300.search import GridSearch
from pytorchsph_gb300.serve import SceneBatch, SceneSpec
from pytorchsph_gb300.sim import SimConfig, Simulation

G = 9.81


def listed():
    return [
        # An interactive or test-sized scene searched on its own: a call with its host waits,
        # where launches and latency are all there is.
        {"name": "search_2k", "kind": "search", "n": 2025, "layout": "lattice", "ratio": 1, "sync": True},
        # The search + density benchmark, evenly spread particles, capacities given and no host wait.
        {"name": "search_1m", "kind": "search", "n": 1 << 20, "layout": "lattice", "ratio": 1, "sync": False},
        # The same with half the particles in a dense cluster (rows of very different lengths),
        # grid cells of half a support as the tuner picks for it.
        {"name": "search_blob_1m", "kind": "search", "n": 1000003, "layout": "blob", "ratio": 2, "sync": False},
        # neighborSearchModule.search as the reference's solver drivers call it every step:
        # (i, j)-ordered pairs, unit vectors and distances.
        {"name": "module_search_260k", "kind": "coo", "n": 260017},
        # The reference's constructNeighborhoodsCUDA over its extension functions.
        {"name": "extension_65k", "kind": "extension", "n": 65537},
        # One deltaSPH timestep of the reference's driver with this package's modules, walls included.
        {"name": "modules_30k", "kind": "modules", "nx": 173, "ny": 177},
        # Ten steps of a small tank, one captured graph per step: launch latency.
        {"name": "steps_8k", "kind": "steps", "nx": 128, "ny": 64, "integration": "semiImplicitEuler",
         "diffusion": "deltaSPH", "steps": 10},
        # A mid-sized tank with the fourth-order integrator (four right-hand sides a step).
        {"name": "steps_rk4_150k", "kind": "steps", "nx": 613, "ny": 251, "integration": "RK4", "diffusion": "MOG",
         "steps": 2},
        # The DFSPH right-hand side of the dam-break benchmark's block, close to settled: search,
        # both pressure solves, viscosity.
        {"name": "dfsph_262k", "kind": "dfsph", "nx": 512, "ny": 512, "dt": 5e-4, "fill": 0.99},
        # The serving batch: dam breaks and drops of the request trace's sizes, stepped together.
        {"name": "serve_100", "kind": "serve", "scenes": 100, "n_min": 2048, "n_max": 131072, "steps": 5},
        # Training-like use: a float32 rollout of the drop and its gradient.
        {"name": "drop_f32_16k", "kind": "drop", "n": 16384, "steps": 20, "fp64": False},
        # The same in double precision, as gradients are validated.
        {"name": "drop_f64_4k", "kind": "drop", "n": 4096, "steps": 10, "fp64": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search", "search", "coo", "extension", "modules", "steps", "dfsph", "serve", "drop"])
    if kind == "search":
        return {"kind": kind, "n": _log(rng, 1500, 1 << 20), "layout": rng.choice(["lattice", "blob"]),
                "ratio": rng.choice([1, 2]), "sync": rng.random() < 0.5}
    if kind == "coo":
        return {"kind": kind, "n": _log(rng, 1500, 260000)}
    if kind == "extension":
        return {"kind": kind, "n": _log(rng, 1500, 65000)}
    if kind == "serve":
        lo = _log(rng, 2048, 32768)
        return {"kind": kind, "scenes": _log(rng, 2, 90), "n_min": lo, "n_max": lo * rng.choice([1, 2, 4]), "steps": 5}
    if kind == "drop":
        fp64 = rng.random() < 0.4
        return {"kind": kind, "n": _log(rng, 1000, 4000 if fp64 else 16000), "steps": rng.randint(4, 10 if fp64 else 20),
                "fp64": fp64}
    n = _log(rng, 2000, {"modules": 30000, "steps": 150000, "dfsph": 260000}[kind])
    nx = max(16, int(math.sqrt(n * rng.uniform(0.5, 2.0))))
    c = {"kind": kind, "nx": nx, "ny": max(16, n // nx)}
    if kind == "steps":
        rk4 = rng.random() < 0.4
        c.update(integration="RK4" if rk4 else "semiImplicitEuler", diffusion=rng.choice(["MOG", "deltaSPH"]),
                 steps=2 if rk4 else 10)
    if kind == "dfsph":
        c.update(dt=rng.choice([2e-4, 5e-4, 1e-3]), fill=round(rng.uniform(0.97, 1.0), 4))
    return c


# ------------------------------------------------------------------------------ inputs
def _points(case, seed):
    """Positions, supports and areas of a search case in [0, 1]^2: support 3 dx, areas around
    dx^2.  The seed draws the areas and where the numbering of the particles begins, so that
    every seed has the same pairs between other particles, and buffers of the same size."""
    n = case["n"]
    side = math.ceil(math.sqrt(n))
    if case.get("layout") == "blob":
        pos = workloads.gaussian_uniform_mix(n, 0.1, (0.5, 0.5), 0)
    else:
        pos = workloads.jittered_lattice(side, 0.1, 0)[:n]
    dx = 1.0 / side
    rng = np.random.default_rng(seed)
    pos = torch.from_numpy(np.roll(pos, int(rng.integers(1, n)), axis=0)).cuda()
    area = torch.from_numpy((dx * dx * rng.uniform(0.9, 1.1, n)).astype(np.float32)).cuda()
    return pos, torch.full((n,), 3.0 * dx, device="cuda"), area, float(np.float32(3.0 * dx))


def _tank(case, seed):
    """A sloshing pool: a block of nx x ny particles that fills the tank's width (the block of a
    dam break for the modules), with jittered positions, the velocity of a standing wave and
    small density deviations.  DFSPH takes `fill` times the lattice's particle area: below 1 a
    settled fluid, whose pressure solve ends after a few sweeps, at 1 the start of a dam
    break, which runs to the sweep limit."""
    nx, ny = case["nx"], case["ny"]
    dfsph = case["kind"] == "dfsph"
    dx = 0.002 if dfsph else 0.01
    tank = (4 * nx * dx if case["kind"] == "modules" else nx * dx, 1.5 * ny * dx)
    sc = workloads.dam_break(nx, ny, dx, tank)
    rng = np.random.default_rng(seed)
    n = len(sc["pos"])
    jitter = 0.05 * dx if dfsph else 0.02 * dx
    sc["pos"] = (sc["pos"] + rng.uniform(-jitter, jitter, (n, 2))).astype(np.float32)
    x, y, k = sc["pos"][:, 0], sc["pos"][:, 1], np.pi / (nx * dx)
    wave = np.stack([np.sin(k * x) * np.cosh(k * y), -np.cos(k * x) * np.sinh(k * y)], 1) / np.cosh(k * ny * dx)
    sc["vel"] = (rng.uniform(0.2, 0.4) * wave + rng.uniform(-0.01, 0.01, (n, 2))).astype(np.float32)
    sc["rho"] = (1.0 + rng.uniform(0.0, 1e-3, n)).astype(np.float32)
    sc["area"] = (sc["area"] * case.get("fill", 1.0)).astype(np.float32)
    return sc, float(10.0 * np.sqrt(2 * G * sc["column_height"]))


def _tank_config(case, sc, c0):
    if case["kind"] == "dfsph":
        return SimConfig(solver="dfsph", dt=case["dt"], c0=c0)
    return SimConfig(solver="deltaSPH", integration=case["integration"], dt=0.1 * sc["h"] / c0, c0=c0,
                     density_diffusion=case["diffusion"])


def _requests(case, seed):
    rng = np.random.default_rng(seed)
    specs = []
    # Sizes and aspects are spread evenly over their ranges, so that every seed has the same
    # work; the seed draws the drops' amplitudes and the particles' places.
    for k, s in enumerate(np.exp(np.linspace(math.log(case["n_min"]), math.log(case["n_max"]), case["scenes"]))):
        req = {"n": int(s), "kind": "dam_break" if k % 2 == 0 else "drop",
               "shape": 0.5 + 1.5 * (0.618 * k % 1.0) if k % 2 == 0 else float(rng.uniform(0.5, 2.0))}
        sc, p = workloads.make_request_scene(req)
        sc["pos"] = (sc["pos"] + rng.uniform(-0.02 * sc["dx"], 0.02 * sc["dx"], sc["pos"].shape)).astype(np.float32)
        specs.append(SceneSpec(sc, SimConfig(dt=p["dt"], c0=p["c0"], density_diffusion=p["diffusion"],
                                             gravity=p["gravity"], point_source=p["point_source"])))
    return specs


def _drop(case, seed):
    sc = workloads.oscillating_drop(case["n"], 0.5, 0.8)
    rng = np.random.default_rng(seed)
    dt = torch.float64 if case["fp64"] else torch.float32
    dx = sc["dx"]
    sc["pos"] = (sc["pos"] + rng.uniform(-0.02 * dx, 0.02 * dx, sc["pos"].shape)).astype(np.float32)
    v0 = torch.from_numpy(sc["vel"] + rng.normal(0, 0.01, sc["vel"].shape)).to("cuda", dt)
    # a loss that asks for a smaller oscillation, as fitting the viscosity does
    grad = torch.from_numpy((sc["vel"] + rng.normal(0, 0.05, sc["vel"].shape)) / len(v0)).to("cuda", dt)
    return sc, v0, grad


def _module_config(sc, c0):
    return {"particle": {"support": sc["h"], "packing": 0.4},
            "fluid": {"restDensity": 1000.0, "c0": c0, "backgroundPressure": False},
            "pressure": {"gamma": 7.0, "kappa": 1.0, "fluidPressureTerm": "TaitEOS", "boundaryPressureTerm": "PBSPH"},
            "diffusion": {"alpha": 0.01, "delta": 0.1, "kinematic": 0.01, "boundaryDiffusion": True,
                          "densityScheme": "deltaSPH"},
            "compute": {"precision": torch.float32, "device": "cuda", "maxNeighbors": 256},
            "neighborSearch": {"gradientThreshold": 1e-7, "supportScale": 1.0, "sortNeighborhoods": True},
            "domain": {"virtualMin": [float(v) for v in sc["vmin"]], "virtualMax": [float(v) for v in sc["vmax"]]},
            "simulation": {"densityScheme": "continuum", "scheme": "deltaSPH", "boundaryScheme": "solid",
                           "bodyForces": True},
            "gravity": {"magnitude": G, "direction": [0.0, -1.0], "pointSource": False, "potentialField": True,
                        "center": [0.0, 0.0]},
            "solidBoundary": {"recomputeBoundary": False, "layers": 3}}


class _Driver:
    """The attributes of a simulation object that the modules read, and its timestep order."""

    def __init__(self, sc, c0):
        cuda = lambda a: torch.as_tensor(np.asarray(a, np.float32), device="cuda").contiguous()
        self.state = {"fluidPosition": cuda(sc["pos"]), "fluidVelocity": cuda(sc["vel"]),
                      "fluidDensity": cuda(sc["rho"]), "fluidArea": cuda(sc["area"]),
                      "fluidSupport": cuda(sc["support"]), "numParticles": len(sc["pos"])}
        cfg = _module_config(sc, c0)
        self.neighborSearch = modules.neighborSearchModule()
        self.boundaryModule = modules.solidBoundaryModule()
        self.densityDiffusionModule = modules.densityDiffusionModule()
        self.density, self.gravity, self.momentum = (modules.densityModule(), modules.gravityModule(),
                                                     modules.momentumModule())
        self.pressure, self.viscosity, self.laminar = (modules.pressureModule(), modules.diffusionModule(),
                                                       modules.laminarViscosityModule())
        self.modules = [self.neighborSearch, self.boundaryModule, self.densityDiffusionModule, self.density,
                        self.gravity, self.momentum, self.pressure, self.viscosity, self.laminar]
        for m in self.modules:
            for p in m.getParameters() or []:
                p.parseConfig(cfg)
            m.initialize(cfg, self.state)
        self.boundaryModule.setWalls(cuda(sc["wall_pos"]), cuda(sc["ghost_pos"]), cuda(sc["wall_area"]))

    def sync(self, t):
        return

    def timestep(self):
        st = self.state
        for m in self.modules:
            m.resetState(st)
        self.neighborSearch.search(st, self)
        self.boundaryModule.boundaryNeighborhoodSearch(st, self)
        self.density.evaluate(st, self)
        self.boundaryModule.evalBoundaryDensity(st, self)
        st["fluidAcceleration"] = torch.zeros_like(st["fluidVelocity"])
        self.gravity.evaluate(st, self)
        self.momentum.computeDpDt(st, self)
        self.densityDiffusionModule.computeDensityDiffusion(st, self)
        self.pressure.computePressure(st, self)
        self.pressure.computePressureAcceleration(st, self)
        self.viscosity.evaluate(st, self)
        self.laminar.computeLaminarViscosity(st, self)
        return [st["fluidAcceleration"], st["dpdt"], st["fluidPressure"], self.boundaryModule.boundaryDensity]


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind in ("search", "coo", "extension"):
        s["pos"], s["support"], s["area"], s["h"] = _points(case, seed)
        s["lo"], s["hi"] = np.zeros(2, np.float32), np.ones(2, np.float32)
    if kind == "search":
        s["engine"] = GridSearch(cell_ratio=case["ratio"])
        s["caps"] = {}
        if not case["sync"]:
            # a program that does not wait for each search sizes its buffers from a first one
            r = s["engine"].run(s["pos"], s["support"], s["area"], kernel_support=s["h"], min_coord=s["lo"],
                                max_coord=s["hi"])
            s["caps"] = {"cell_capacity": r.cell_capacity, "pair_capacity": r.num_pairs, "sync": False}
    elif kind == "coo":
        m = modules.neighborSearchModule()
        cfg = {"particle": {"support": s["h"]}, "compute": {"maxNeighbors": 256, "precision": torch.float32,
                                                            "device": "cuda"},
               "domain": {"virtualMin": [0.0, 0.0], "virtualMax": [1.0, 1.0]}}
        for p in m.getParameters():
            p.parseConfig(cfg)
        m.initialize(cfg, None)
        s["module"] = m
        s["state"] = {"fluidPosition": s["pos"], "fluidSupport": s["support"]}
    elif kind == "modules":
        s["driver"] = _Driver(*_tank(case, seed))
    elif kind in ("steps", "dfsph"):
        sc, c0 = _tank(case, seed)
        s["sim"] = Simulation(sc, _tank_config(case, sc, c0))
        if kind == "steps":
            # the first step sizes the neighbor buffer; the next ones replay it as one graph
            s["sim"].step()
            s["sim"].capture()
    elif kind == "serve":
        s["batch"] = SceneBatch(_requests(case, seed))
        s["batch"].capture()
    elif kind == "drop":
        sc, v0, grad = _drop(case, seed)
        s["rollout"] = DropRollout(sc, 10.0, 0.1 * sc["h"] / 10.0, fp64=case["fp64"])
        s["v0"], s["grad"] = v0.requires_grad_(), grad
        s["alpha"] = torch.tensor(0.01, dtype=torch.float64, device="cuda", requires_grad=True)
    return s


def _by_particle(sim, fields):
    """Fields of a Simulation, which keeps its rows sorted by cell, in particle order."""
    uid = sim.arr["uid"].long()
    return [torch.empty_like(f).index_copy_(0, uid, f) for f in fields]


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "search":
        r = s["engine"].run(s["pos"], s["support"], s["area"], kernel_support=s["h"], min_coord=s["lo"],
                            max_coord=s["hi"], **s["caps"])
        return [r.density(), r.order[:r.n], r.offsets, r.cols]
    if kind == "coo":
        return list(s["module"].search(s["state"], None))
    if kind == "extension":
        i, j, _, _, (_, _, order, _, _), (table, _), (cells, _, _, _) = neighborhoods.constructNeighborhoodsCUDA(
            s["pos"], s["support"], minCoord=s["lo"], maxCoord=s["hi"])
        return [i, j, order, table, cells]
    if kind == "modules":
        return s["driver"].timestep()
    if kind == "steps":
        sim = s["sim"]
        for _ in range(case["steps"]):
            sim.step(sync=False)
        return _by_particle(sim, [sim.arr["x"], sim.arr["v"], sim.arr["rho"]])
    if kind == "dfsph":
        sim = s["sim"]
        acc, _, _ = sim.rhs()
        return _by_particle(sim, [acc, sim.last["pressure"], sim.arr["rho"]]) + [sim.last["divergence_iters"],
                                                                                sim.last["density_iters"]]
    if kind == "serve":
        b = s["batch"]
        for _ in range(case["steps"]):
            b.step()
        out = b.states_device()
        return [out["x"], out["v"], out["rho"]]
    x = drop_rollout(s["rollout"], s["v0"], s["alpha"], case["steps"])
    gv, ga = torch.autograd.grad(x, [s["v0"], s["alpha"]], s["grad"])
    return [x.detach(), gv, ga]


def work(case):
    """Bytes: each input read and each output written once.  Flops: the pair terms' arithmetic."""
    kind = case["kind"]
    n = case["n"] if "n" in case else case["nx"] * case["ny"] if "nx" in case else 0
    pairs = 28.3 * n
    if case.get("layout") == "blob":
        pairs *= 0.75 + math.ceil(math.sqrt(n)) ** 2 / n / (16 * math.pi * 0.01)
    if kind == "search":
        return {"bytes": n * (16 + 4 + 4 + 4) + 4 * pairs, "flops": 20 * pairs}
    if kind == "coo":
        return {"bytes": 12 * n + 28 * pairs, "flops": 12 * pairs}
    if kind == "extension":
        return {"bytes": n * (12 + 8 + 8) + 16 * pairs, "flops": 6 * pairs}
    if kind == "modules":
        return {"bytes": n * (8 + 8 + 12 + 16), "flops": 120 * pairs}
    if kind == "steps":
        rhs = case["steps"] * (4 if case["integration"] == "RK4" else 1)
        return {"bytes": n * 44 * case["steps"], "flops": 90 * pairs * rhs}
    if kind == "dfsph":
        return {"bytes": n * (24 + 16), "flops": 2 * 3 * 40 * pairs}
    if kind == "serve":
        n = float(np.exp(np.linspace(math.log(case["n_min"]), math.log(case["n_max"]), case["scenes"])).sum())
        return {"bytes": n * 44 * case["steps"], "flops": 100 * 28.3 * n * case["steps"]}
    w = 8 if case["fp64"] else 4
    return {"bytes": n * w * (6 + 2 + 4), "flops": case["steps"] * pairs * (70 + 70 + 300)}


# ------------------------------------------------------------------------------ 64 bits
def _pairs(xa, h, xb):
    """Pairs (a, b) in order with the distance of the float32 positions below h."""
    cell = float(h) * 1.0001
    lo = torch.minimum(xa.min(0).values, xb.min(0).values).double() - cell
    ca, cb = (((t.double() - lo) / cell).floor().long() for t in (xa, xb))
    nx = int(max(ca[:, 0].max(), cb[:, 0].max())) + 3
    key, order = (cb[:, 0] + 1 + nx * cb[:, 1]).sort(stable=True)
    rows, cols = [], []
    for dy in (-1, 0, 1):
        k = ca[:, 0] + 1 + nx * (ca[:, 1] + dy)
        b, e = torch.searchsorted(key, k - 1), torch.searchsorted(key, k + 1, right=True)
        num = e - b
        i = torch.repeat_interleave(torch.arange(len(xa), device=xa.device), num)
        j = order[torch.arange(len(i), device=xa.device) - (num.cumsum(0) - num)[i] + b[i]]
        d = xa[i] - xb[j]
        # sqrt(fma(dx, dx, dy dy)) in float32, as the reference compares it
        r = (d[:, 0].double() ** 2 + (d[:, 1] * d[:, 1]).double()).float().sqrt()
        keep = r < torch.tensor(h, dtype=torch.float32, device=r.device)
        rows.append(i[keep])
        cols.append(j[keep])
    i, j = torch.cat(rows), torch.cat(cols)
    k = (i * len(xb) + j).sort().values
    return k // len(xb), k % len(xb)


def _sum(v, i, n):
    return torch.zeros((n,) + v.shape[1:], dtype=v.dtype, device=v.device).index_add_(0, i, v)


def _dot(a, b):
    return (a * b).sum(-1)


class _Geo:
    """Pair geometry d = x_i - x_j with the Wendland kernel and gradient and the spiky gradient."""

    def __init__(self, d, h):
        r2 = _dot(d, d)
        self.far = r2 >= 1e-14
        self.r = torch.where(self.far, r2, torch.ones_like(r2)).sqrt() * self.far
        q = self.r / h
        self.d, self.q, self.r2 = d, q, r2
        self.w = (1 - q) ** 4 * (1 + 4 * q) * 7 / (math.pi * h ** 2)
        self.g = (-140 / (math.pi * h ** 4) * (1 - q) ** 3 * self.far)[:, None] * d
        e = d / torch.where(self.far, self.r, torch.ones_like(q))[:, None] * self.far[:, None]
        self.e = e
        self.spiky = -30 / (math.pi * h ** 3) * ((1 - q) ** 2)[:, None] * e


def _cfg(h, c0, alpha=0.01, nu=0.001, diffusion="deltaSPH", gravity=(0.0, -G), point=False):
    return {"h": h, "c0": c0, "alpha": alpha, "nu": nu, "diffusion": diffusion, "gravity": gravity, "point": point}


def _walls(sc):
    if not len(sc["wall_pos"]):
        return None
    return {k: torch.from_numpy(sc[n]).cuda() for k, n in (("x", "wall_pos"), ("ghost", "ghost_pos"), ("A", "wall_area"))}


def _tait(rt, c):
    return 1000.0 * c["c0"] ** 2 / 7.0 * (rt ** 7 - 1)


def _mdbc(x, A, V, W, c):
    """Wall densities from the fluid around the walls' ghost points."""
    b, j = _pairs(W["ghost"], c["h"], x.detach().float())
    nb, xg = len(W["x"]), W["ghost"].double()
    g = _Geo(xg[b] - x[j], c["h"])
    one = torch.cat([torch.ones_like(g.w)[:, None], -g.d], 1)
    left = torch.cat([g.w[:, None], g.g], 1)
    M = _sum((V[j, None, None] * left[:, :, None] * one[:, None, :]).reshape(-1, 9), b, nb).reshape(-1, 3, 3)
    rhs = _sum(1000.0 * A[j, None] * left, b, nb)
    cnt = torch.bincount(b, minlength=nb)
    rho = torch.where(cnt > 0, rhs[:, 0] / M[:, 0, 0] / 1000.0, torch.ones_like(rhs[:, 0]))
    full = cnt > 10
    s = (torch.linalg.pinv(M[full].cpu()).cuda() @ rhs[full][:, :, None])[:, :, 0]
    rho[full] = (s[:, 0] + _dot(W["x"].double()[full] - xg[full], s[:, 1:])) / 1000.0
    return rho.clamp(min=1.0)


def _rhs(x, v, rt, A, W, c, extras=None):
    """deltaSPH: acceleration and density rate of a scene (src/deltaSPH.py's timestep)."""
    h, n, eps = c["h"], len(x), 0.1 * c["h"] ** 2
    x32 = x.detach().float()
    i, j = _pairs(x32, h, x32)
    g = _Geo(x[i] - x[j], h)
    rho, V, p = 1000.0 * rt, A / rt, _tait(rt, c)
    u, r2 = v[j] - v[i], g.r2 + eps
    rg = -_dot(g.d, g.g)
    diff = h * 0.1 * c["c0"]
    dp = -_sum(_dot(u, g.g) * V[j] * rho[j], i, n)
    acc = -_sum(((p[i] + p[j]) * V[j])[:, None] * g.g, i, n) / rho[:, None]
    pij = (-_dot(u, g.d)).clamp(max=0) / r2
    acc = acc + h * c["alpha"] * c["c0"] * _sum((pij * V[j] * rho[j] / (rho[i] + rho[j]))[:, None] * g.g, i, n)
    lam = 8 * rho[j] * V[j] * rho[i] * c["nu"] * rg / ((rho[i] + rho[j]) ** 2 * r2)
    acc = acc + _sum(lam[:, None] * u, i, n)
    acc = acc - x if c["point"] else acc + torch.tensor(c["gravity"], dtype=x.dtype, device=x.device)
    if W is not None:
        rb = _mdbc(x, A, V, W, c)
        Vb, pb, xb = W["A"].double() / rb, _tait(rb, c), W["x"].double()
        b, f = _pairs(W["x"], h, x32)
        gb = _Geo(x[f] - xb[b], h)
        rhob = 1000.0 * rb
        ud = -v[f]
        dp = dp - _sum(_dot(ud, gb.g) * Vb[b] * rhob[b], f, n)
        acc = acc - _sum(((p[f] + pb[b]) * Vb[b])[:, None] * gb.g, f, n) / rho[:, None]
        pib = (-_dot(ud, gb.d)).clamp(max=0) / (gb.r2 + eps)
        acc = acc + h * c["alpha"] * c["c0"] * _sum((pib * Vb[b] * rhob[b] / (rho[f] + rhob[b]))[:, None] * gb.g, f, n)
        if extras is not None:
            extras["wall_rho"] = rb
    first = 2 * (rho[j] - rho[i]) / r2 * rg * V[j]
    if c["diffusion"] == "MOG":
        return acc, dp + diff * _sum(first, i, n)
    L = -_sum((V[j, None, None] * g.d[:, :, None] * g.g[:, None, :]).reshape(-1, 4), i, n)
    s = _sum((2 * (rho[j] - rho[i]) * V[j])[:, None] * g.g, i, n)
    if W is not None:
        L = L - _sum((Vb[b, None, None] * gb.d[:, :, None] * gb.g[:, None, :]).reshape(-1, 4), f, n)
        s = s + _sum((2 * (rhob[b] - rho[f]) * Vb[b])[:, None] * gb.g, f, n)
    det = L[:, 0] * L[:, 3] - L[:, 1] * L[:, 2]
    gr = -torch.stack([L[:, 3] * s[:, 0] - L[:, 1] * s[:, 1], L[:, 0] * s[:, 1] - L[:, 2] * s[:, 0]], 1) / det[:, None]
    return acc, dp + diff * _sum(first - _dot(gr[i] + gr[j], g.g) * V[j], i, n)


def _euler(x, v, rt, A, W, c, dt):
    acc, dp = _rhs(x, v, rt, A, W, c)
    v1 = v + dt * acc
    return x + dt * v1, v1, rt + dt * dp / 1000.0


def _rk4(x, v, rt, A, W, c, dt):
    k, s = [], (x, v, rt)
    for a in (0.5, 0.5, 1.0, None):
        acc, dp = _rhs(*s, A, W, c)
        k.append((s[1], acc, dp / 1000.0))
        if a:
            s = tuple(y + a * dt * d for y, d in zip((x, v, rt), k[-1]))
    return tuple(y + dt / 6 * (a + 2 * b + 2 * d + e) for y, a, b, d, e in zip((x, v, rt), *k))


def _dfsph(sc, dt, c0):
    """DFSPH: acceleration, pressure and density of a scene (src/dfsph.py's timestep)."""
    x32 = torch.from_numpy(sc["pos"]).cuda()
    x, u, A = x32.double(), torch.from_numpy(sc["vel"]).cuda().double(), torch.from_numpy(sc["area"]).cuda().double()
    W, h, n = _walls(sc), sc["h"], len(x32)
    xb, Ab = W["x"].double(), W["A"].double()
    nb = len(xb)
    i, j = _pairs(x32, h, x32)
    b, f = _pairs(W["x"], h, x32)
    g, gb = _Geo(x[i] - x[j], h), _Geo(xb[b] - x[f], h)
    wi, wj = _pairs(W["x"], h, W["x"])
    rt = _sum(g.w * A[j], i, n)
    V = A / rt
    rb = (_sum(_Geo(xb[wi] - xb[wj], h).w * Ab[wj], wi, nb) + _sum(gb.w * A[f], b, nb)).clamp(max=1.0)
    rt = rt + _sum(gb.w * Ab[b], f, n)
    rho, rhob, m = 1000.0 * rt, 1000.0 * rb, 1000.0 * A
    Aa, Ba = A / rt, Ab / rb
    acc = torch.tensor([0.0, -G], dtype=x.dtype, device=x.device).expand(n, 2)
    iters, S, Sb = [], g.spiky, gb.spiky
    for density, limit in ((False, 1e-3), (True, 1e-4)):
        vs = u + dt * acc
        k1 = _sum(Aa[j, None] * S, i, n)
        k2 = _sum(Aa[j] ** 2 / m[j] * _dot(S, S), i, n)
        src = -dt * _sum(Aa[j] * _dot(vs[i] - vs[j], S), i, n)
        if density:
            k1 = k1 + _sum(Ba[b, None] * Sb, f, n)
            k2 = k2 + _sum(Ba[b] ** 2 / (1000.0 * Ab[b]) * _dot(Sb, Sb), f, n)
            src = 1 - rt + src + dt * _sum(Ba[b] * _dot(vs[f], Sb), f, n)
            walpha = (-dt ** 2 * Ba * _sum(Aa[f] ** 2 / m[f] * _dot(Sb, Sb), b, nb)).clamp(max=-1e-4 * h * h)
            wsrc = 1 - rb + dt * _sum(Aa[f] * _dot(vs[f], Sb), b, nb)
        alpha = (-dt ** 2 * Aa / m * _dot(k1, k1) - dt ** 2 * Aa * k2).clamp(-1.0, -1e-7)
        p, pb, err, it = torch.zeros_like(A), torch.zeros_like(Ab), 0.0, 0

        def accel():
            a = -_sum((m[j] * (p[i] / rho[i] ** 2 + p[j] / rho[j] ** 2))[:, None] * S, i, n)
            if density:
                a = a + _sum((1000.0 * Ab[b] * (p[f] / rho[f] ** 2 + pb[b] / rhob[b] ** 2))[:, None] * Sb, f, n)
            return a

        while (it < 2 or err > limit) and it <= 100:
            a = accel()
            ks = dt ** 2 * _sum(Aa[j] * _dot(a[i] - a[j], S), i, n)
            if density:
                bks = -dt ** 2 * _sum(Aa[f] * _dot(a[f], Sb), b, nb)
                ks = ks - dt ** 2 * _sum(Ba[b] * _dot(a[f], Sb), f, n)
                wres = bks - wsrc
                pb = (pb - 0.5 * wres / walpha).clamp(min=0.0)
            res = ks - src
            p = p - 0.3 * res / alpha
            total, count = res.clamp(min=-limit).sum(), n
            if density:
                p = p.clamp(min=0.0)
                total, count = total + wres.clamp(min=-limit).sum(), n + nb
            err, it = float(total) / count, it + 1
        acc = acc + accel()
        iters.append(it)
    eps, ud = 0.1 * h * h, u[j] - u[i]
    r2, mj = g.r2 + eps, rho[j] * V[j]
    visc = (-_dot(ud, g.d)).clamp(max=0) / r2 * mj / (rho[i] + rho[j])
    lam = 8 * mj * rho[i] * 0.001 * -_dot(g.d, g.g) / ((rho[i] + rho[j]) ** 2 * r2)
    rb2 = gb.r2 + eps
    wv = (-_dot(u[f], gb.d)).clamp(max=0) / rb2 * 1000.0 * Ab[b] / (rho[f] + rhob[b])
    vk = h * 0.01 * c0
    acc = acc + vk * _sum(visc[:, None] * g.g, i, n) - vk * _sum(wv[:, None] * gb.g, f, n) + _sum(lam[:, None] * ud, i, n)
    return [acc, p, rt, None, None]


def exact(case, seed):
    kind = case["kind"]
    if kind == "search":
        x32, _, area, h = _points(case, seed)
        i, j = _pairs(x32, h, x32)
        x = x32.double()
        return [_sum(_Geo(x[i] - x[j], h).w * area[j].double(), i, len(x)), None, None, None]
    if kind == "coo":
        x32, _, _, h = _points(case, seed)
        i, j = _pairs(x32, h, x32)
        g = _Geo((x32[i].double() - x32[j].double()), h)
        return [None, g.e, g.q]
    if kind == "extension":
        return None
    if kind == "dfsph":
        sc, c0 = _tank(case, seed)
        return _dfsph(sc, case["dt"], c0)
    cuda = lambda a: torch.from_numpy(a).cuda().double()
    if kind == "drop":
        sc, v0, grad = _drop(case, seed)
        x, A, rt = cuda(sc["pos"]), cuda(sc["area"]), cuda(sc["rho"])
        v0 = v0.double().requires_grad_()
        alpha = torch.tensor(0.01, dtype=torch.float64, device="cuda", requires_grad=True)
        c = _cfg(sc["h"], 10.0, alpha=alpha, diffusion="MOG", point=True)
        v, dt = v0, 0.1 * sc["h"] / 10.0
        for _ in range(case["steps"]):
            x, v, rt = _euler(x, v, rt, A, None, c, dt)
        gv, ga = torch.autograd.grad(x, [v0, alpha], grad.double())
        return [x.detach(), gv, ga]
    if kind in ("modules", "steps"):
        sc, c0 = _tank(case, seed)
        s, A, W = (cuda(sc["pos"]), cuda(sc["vel"]), cuda(sc["rho"])), cuda(sc["area"]), _walls(sc)
        if kind == "modules":
            c, extra = _cfg(sc["h"], c0, nu=0.01), {}
            acc, dp = _rhs(*s, A, W, c, extra)
            return [acc, dp, _tait(s[2], c), extra["wall_rho"]]
        c = _cfg(sc["h"], c0, diffusion=case["diffusion"])
        dt = float(np.float32(0.1 * sc["h"] / c0))
        step = _rk4 if case["integration"] == "RK4" else _euler
        for _ in range(case["steps"] + 1):   # prepare takes the first
            s = step(*s, A, W, c, dt)
        return list(s)
    out = []
    for sp in _requests(case, seed):
        sc, cfg = sp.scene, sp.cfg
        s, A, W = (cuda(sc["pos"]), cuda(sc["vel"]), cuda(sc["rho"])), cuda(sc["area"]), _walls(sc)
        c = _cfg(sc["h"], cfg.c0, gravity=cfg.gravity, point=cfg.point_source)
        for _ in range(case["steps"] + 1):
            s = _euler(*s, A, W, c, float(np.float32(cfg.dt)))
        out.append(s)
    return [torch.cat(t) for t in zip(*out)]
