"""DFSPH with the pairs from the cell rows (neighbor lists of the density pass, several lanes per
particle) against the same right-hand side over the CSR list (one thread per row): the numbers
of particles where the lanes per particle change, and a block so dense that the lists overflow
and the cell rows are tested again.  Both sum the same float32 terms in different orders: a sum
of ~30 terms is off by at most 2e-6 of its largest term, a few sweeps carry that to 2e-5 of the
field's maximum; the bar is 1e-4, with equal iteration counts."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a.double() - b.double()).abs().max() / max(float(b.double().abs().max()), 1e-30))


@pytest.mark.parametrize("nx,ny,squeeze", [(5, 3, 1.0), (90, 91, 1.0), (91, 91, 1.0), (181, 181, 1.0),
                                           (182, 182, 1.0), (443, 443, 1.0), (444, 444, 1.0), (40, 40, 0.5)])
def test_lists_match_csr(cuda, nx, ny, squeeze):
    from pytorchsph_gb300 import workloads
    from pytorchsph_gb300.sim import SimConfig, Simulation
    dx = 0.01
    sc = workloads.dam_break(nx, ny, dx, (nx * dx * 1.5, ny * dx * 1.5))
    rng = np.random.default_rng(nx)
    sc["pos"] = ((sc["pos"] + rng.uniform(-0.05 * dx, 0.05 * dx, sc["pos"].shape)) * squeeze).astype(np.float32)
    sc["vel"] = rng.uniform(-0.2, 0.2, sc["pos"].shape).astype(np.float32)
    sc["area"] = (sc["area"] * 0.98).astype(np.float32)
    cfg = SimConfig(solver="dfsph", dt=5e-4, max_density_iters=4, max_divergence_iters=4)
    got = {}
    for pairs in ("cells", "csr"):
        sim = Simulation(sc, cfg, cuda, pairs=pairs)
        acc, _, _ = sim.rhs()
        order = torch.argsort(sim.arr["uid"].long())
        got[pairs] = [t[order] for t in (acc, sim.last["pressure"], sim.last["alpha"], sim.arr["rho"])] + [
            sim.dfsph_arrays["wall_pressure"].clone(), sim.dfsph_arrays["wall_rho"].clone()]
        got[pairs + "_iters"] = (int(sim.last["divergence_iters"]), int(sim.last["density_iters"]))
        assert int(sim.status.item()) == 0
    assert got["cells_iters"] == got["csr_iters"]
    for a, b in zip(got["cells"], got["csr"]):
        assert rel(a, b) < 1e-4
    assert torch.equal(got["cells"][3], got["csr"][3])   # the density sum keeps its order
