"""Objects that a caller's program puts in place of this package's own: what was taken as a
neighbor search stays one."""
import numpy as np
import pytest
import torch

import test_modules_walls_gpu as walls

pytestmark = pytest.mark.gpu


class Delegate:
    """A search that hands out another one's methods."""

    def __init__(self, inner):
        self.search, self.searchExisting = inner.search, inner.searchExisting


class Counted:
    """A search with a searchExisting of its own."""

    def __init__(self, inner):
        self.inner, self.calls = inner, 0
        self.search = inner.search

    def searchExisting(self, *args, **kw):
        self.calls += 1
        return self.inner.searchExisting(*args, **kw)


def wall_lists(cuda, wrap):
    from pytorchsph_gb300 import modules as M, workloads
    sc = workloads.dam_break(12, 16, 0.01, (0.4, 0.3))
    cfg = walls.config(sc, 10.0, "continuum")
    st = walls.state(sc, cuda, sc["rho"])
    sim = walls.Driver()
    inner = M.neighborSearchModule()
    sim.neighborSearch, sim.boundaryModule = wrap(inner), M.solidBoundaryModule()
    walls.setup([inner, sim.boundaryModule], cfg, st)
    t = lambda a: torch.as_tensor(np.asarray(a, np.float32), device=cuda).contiguous()
    sim.boundaryModule.setWalls(t(sc["wall_pos"]), t(sc["ghost_pos"]), t(sc["wall_area"]))
    sim.neighborSearch.search(st, sim)
    sim.boundaryModule.boundaryNeighborhoodSearch(st, sim)
    st["fluidVolume"] = st["fluidArea"]
    sim.boundaryModule.evalBoundaryDensity(st, sim)
    b = sim.boundaryModule
    return [b.boundaryToFluidNeighbors, b.boundaryToFluidNeighborDistances, b.ghostToFluidNeighbors, b._bf.woff,
            b._gf.woff, b.boundaryDensity], sim


@pytest.mark.parametrize("wrap", [Delegate, Counted])
def test_searches_in_place_of_the_module(cuda, wrap):
    want, _ = wall_lists(cuda, lambda inner: inner)
    got, sim = wall_lists(cuda, wrap)
    assert len(want[0][0]) > 0 and all(torch.equal(a, b) for a, b in zip(want, got))
    assert wrap is Delegate or sim.neighborSearch.calls == 2


@pytest.mark.parametrize("more", [1, 3, 4, 12])
@pytest.mark.parametrize("integration", ["semiImplicitEuler", "RK4"])
def test_arrays_added_to_a_simulation(cuda, more, integration):
    """Per-particle arrays of a caller's in sim.arr move with the particles, however many, eagerly and in
    a captured step."""
    from pytorchsph_gb300 import workloads
    from pytorchsph_gb300.sim import SimConfig, Simulation
    sc = workloads.dam_break(20, 15, 0.01, (0.4, 0.3))
    sc["vel"] = np.random.default_rng(1).uniform(-2, 2, sc["pos"].shape).astype(np.float32)
    sim = Simulation(sc, SimConfig(dt=1e-3, c0=10.0, integration=integration, density_diffusion="MOG"), cuda)
    added = {}
    for k in range(more):
        t = torch.arange(sim.n * (1, 2, 4)[k % 3], device=cuda).float().view(sim.n, -1)
        added[f"tracer{k}"] = t
        sim.arr[f"tracer{k}"] = t.clone()
    for _ in range(3):
        sim.step()
    sim.capture()
    for _ in range(3):
        sim.step()
    sim.check()
    uid = sim.arr["uid"].long()
    assert not torch.equal(uid, torch.arange(sim.n, device=cuda))
    for k, t in added.items():
        assert torch.equal(sim.arr[k], t[uid])
    assert sim.steps == 6 and float(sim.time) == pytest.approx(6e-3)


@pytest.mark.parametrize("missing", [None, "_raw_stream", "_device"])
def test_stream_pointer(cuda, missing, monkeypatch):
    """The current stream, also where torch lacks its private short way."""
    from pytorchsph_gb300 import _native as N
    if missing:
        monkeypatch.setattr(N, missing, None)
    side = torch.cuda.Stream(cuda)
    assert N.stream_ptr() == torch.cuda.current_stream().cuda_stream
    with torch.cuda.stream(side):
        assert N.stream_ptr() == side.cuda_stream
