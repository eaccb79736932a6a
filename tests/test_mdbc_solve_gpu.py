"""Wall densities where the 3x3 mDBC system changes its solver and the launch its lanes: tanks whose
support scales the system's condition through the bound between the adjugate and the singular
value sweeps, and batches below and above the walls that get several lanes each.  Against
float64 torch.linalg.pinv with the float32 cut-off (3 FLT_EPSILON) on the same pairs: the float32
sums are off by up to 30 x 6e-8 of their terms, which a system of condition c turns into 2e-6 c of
the density; walls are held to max(1e-5, 2e-6 c) for c up to 1e3, and the others to finite values
of at least 1 (there the float32 reference disagrees with itself)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def expected(sc, rho0=1000.0):
    x, xg, xb = (np.asarray(sc[k], np.float64) for k in ("pos", "ghost_pos", "wall_pos"))
    h, A = float(sc["h"]), np.asarray(sc["area"], np.float64)
    V = A / np.asarray(sc["rho"], np.float64)
    rho, cond = np.ones(len(xb)), np.ones(len(xb))
    for b in range(len(xb)):
        d = (sc["ghost_pos"][b] - sc["pos"]).astype(np.float32)
        r = np.sqrt((d[:, 0].astype(np.float64) ** 2 + (d[:, 1] * d[:, 1]).astype(np.float64)).astype(np.float32))
        j = np.nonzero(r < np.float32(h))[0]
        if len(j) == 0:
            continue
        d = xg[b] - x[j]
        r = np.sqrt((d ** 2).sum(1))
        q = r / h
        w = (1 - q) ** 4 * (1 + 4 * q) * 7 / (np.pi * h ** 2)
        g = (-140 / (np.pi * h ** 4) * (1 - q) ** 3)[:, None] * d
        left = np.concatenate([w[:, None], g], 1)
        M = np.einsum("j,ju,jv->uv", V[j], left, np.concatenate([np.ones((len(j), 1)), -d], 1))
        rhs = rho0 * (A[j, None] * left).sum(0)
        if len(j) > 10:
            s = np.linalg.pinv(M, rcond=3 * np.finfo(np.float32).eps) @ rhs
            rho[b] = (s[0] + (xb[b] - xg[b]) @ s[1:]) / rho0
            cond[b] = np.linalg.cond(M)
        else:
            rho[b] = rhs[0] / M[0, 0] / rho0
    return np.maximum(rho, 1.0), cond


@pytest.mark.parametrize("dx", [0.1, 0.01, 0.002])
def test_wall_density_across_the_solver_bound(cuda, dx):
    from pytorchsph_gb300 import workloads
    from pytorchsph_gb300.sim import SimConfig, Simulation
    sc = workloads.dam_break(13, 11, dx, (20 * dx, 16 * dx))
    rng = np.random.default_rng(3)
    sc["pos"] = (sc["pos"] + rng.uniform(-0.1 * dx, 0.1 * dx, sc["pos"].shape)).astype(np.float32)
    sc["rho"] = (1 + rng.uniform(0, 1e-2, len(sc["pos"]))).astype(np.float32)
    sim = Simulation(sc, SimConfig(dt=1e-6, c0=10.0), cuda)
    sim.rhs()
    got = sim.wall_state()["rho"].astype(np.float64)
    want, cond = expected(sc)
    assert np.isfinite(got).all() and (got >= 1.0).all()
    held = cond <= 1e3
    assert held.sum() > 100
    err = np.abs(got - want)[held] / want[held]
    assert (err <= np.maximum(1e-5, 2e-6 * cond[held])).all(), err.max()


@pytest.mark.parametrize("copies", [1, 40])
def test_batch_walls_match_alone(cuda, copies):
    """40 tanks of 1,188 walls take one lane per wall, a tank alone 16: float32 sums of ~30 terms
    in another order, so within 1e-5 where the system's condition is below 1e3."""
    from pytorchsph_gb300 import workloads
    from pytorchsph_gb300.serve import SceneBatch, SceneSpec
    from pytorchsph_gb300.sim import SimConfig
    sc = workloads.dam_break_scene(2000, 1.0)
    cfg = SimConfig(dt=1e-6, c0=10.0, density_diffusion="deltaSPH")
    batch = SceneBatch([SceneSpec(sc, cfg) for _ in range(copies)], cuda)
    assert (batch.nb > 32768) == (copies == 40)
    batch.step()
    rho = torch.empty_like(batch.w["rho"])
    rho[batch.w["order"].long()] = batch.w["rho"]
    want, cond = expected(sc)
    held = cond <= 1e3
    nb = len(sc["wall_pos"])
    got = rho.cpu().numpy().astype(np.float64).reshape(copies, nb)
    assert (got == got[0]).all()
    assert (np.abs(got[0] - want)[held] <= np.maximum(1e-5, 2e-6 * cond[held]) * want[held]).all()
