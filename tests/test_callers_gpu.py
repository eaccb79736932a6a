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
