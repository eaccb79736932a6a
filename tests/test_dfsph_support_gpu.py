"""DFSPH from the cell rows at supports beyond three spacings: the neighbor lists hold every
particle's and wall's rows, agree with the CSR list, and are no slower than it.

Lists and CSR rows sum the same float32 terms in different orders: 1e-4 of a field's maximum for
fields of a few sweeps, as tests/test_dfsph_lists_gpu.py derives it for sums of 30 terms; a sum
of n terms in another order is off by about sqrt(n) roundings, at 113 terms (6 spacings) twice
as much, 2e-4."""
import numpy as np
import pytest
import torch

from test_dense_sets_gpu import graph_of, time_us
from test_dfsph_lists_gpu import rel

pytestmark = pytest.mark.gpu


def scene(nx, ratio, layers=3):
    from pytorchsph_gb300 import workloads
    dx = 0.01
    sc = workloads.dam_break(nx, nx, dx, (nx * dx * 1.5, nx * dx * 1.5), layers)
    rng = np.random.default_rng(nx)
    n = len(sc["pos"])
    h = np.float32(ratio * dx)
    sc.update(support=np.full(n, h, np.float32), h=float(h), vmin=np.full(2, -2 * h, np.float32),
              vmax=np.float32([nx * dx * 1.5 + 2 * h] * 2))
    sc["pos"] = (sc["pos"] + rng.uniform(-0.05 * dx, 0.05 * dx, (n, 2))).astype(np.float32)
    sc["vel"] = rng.uniform(-0.2, 0.2, (n, 2)).astype(np.float32)
    sc["area"] = (sc["area"] * 0.98).astype(np.float32)
    return sc


def chunk_counts(sim):
    """The particles' and walls' list lengths, the last words of the records (-1: no list)."""
    return sim.dfsph_arrays["records"][-(sim.n + sim.nb):].view(torch.int32)


@pytest.mark.parametrize("nx", [30, 100, 200, 450])   # 8, 4, 2 lanes and 1 lane per particle
@pytest.mark.parametrize("ratio,layers", [(2.0, 3), (3.0, 3), (4.0, 4), (4.5, 5), (6.0, 6)])
def test_lists_hold_the_rows(cuda, nx, ratio, layers):
    from pytorchsph_gb300.sim import SimConfig, Simulation
    sc = scene(nx, ratio, layers)
    cfg = SimConfig(solver="dfsph", dt=5e-4, max_density_iters=4, max_divergence_iters=4)
    got = {}
    for pairs in ("cells", "csr"):
        sim = Simulation(sc, cfg, cuda, pairs=pairs)
        acc, _, _ = sim.rhs()
        order = torch.argsort(sim.arr["uid"].long())
        got[pairs] = [t[order] for t in (acc, sim.last["pressure"], sim.last["alpha"], sim.arr["rho"])] + [
            sim.dfsph_arrays["wall_pressure"].clone(), sim.dfsph_arrays["wall_rho"].clone()]
        if pairs == "cells":
            assert bool((chunk_counts(sim) >= 0).all())
        assert int(sim.status.item()) == 0
    for a, b in zip(got["cells"], got["csr"]):
        assert rel(a, b) < 2e-4


def test_rows_no_list_can_hold(cuda):
    """A support of 20 spacings (1,257 neighbors) runs over the CSR list."""
    from pytorchsph_gb300.sim import SimConfig, Simulation
    sim = Simulation(scene(30, 20.0), SimConfig(solver="dfsph", dt=1e-4), cuda)
    assert sim.pairs == "csr"
    sim.step()
    sim.check()


def test_no_slower_than_csr(cuda):
    from pytorchsph_gb300.sim import SimConfig, Simulation
    took = {}
    for pairs in ("cells", "csr"):
        sim = Simulation(scene(512, 4.5), SimConfig(solver="dfsph", dt=1e-5, max_density_iters=8), cuda, pairs=pairs)
        sim.rhs()
        took[pairs] = time_us(graph_of(lambda: sim.rhs(sync=False)))
    assert took["cells"] < took["csr"], took
