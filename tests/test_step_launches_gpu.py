"""Launches that do two things at once against the two: wall densities beside the records
(particle counts on both sides of the lanes' limits, with and without walls), an RK4 stage against
its sum and update, and the time added by the integrator.  The same operations in the same
order: equal bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(1, 1), (7, 5), (128, 64), (182, 180), (182, 181), (256, 192), (513, 512)])
@pytest.mark.parametrize("diffusion", ["MOG", "deltaSPH"])
@pytest.mark.parametrize("pairs", ["cells", "csr"])
def test_walls_beside_records(cuda, nx, ny, diffusion, pairs):
    from pytorchsph_gb300 import _native as N, workloads
    from pytorchsph_gb300.sim import SimConfig, Simulation, _ref
    sc = workloads.dam_break(nx, ny, 0.01, (max(2 * nx, 8) * 0.01, max(2 * ny, 8) * 0.01))
    rng = np.random.default_rng(nx)
    sc["vel"] = rng.uniform(-0.1, 0.1, sc["pos"].shape).astype(np.float32)
    sim = Simulation(sc, SimConfig(dt=1e-5, c0=10.0, density_diffusion=diffusion), cuda, pairs=pairs)
    acc, _, dpdt = sim.rhs()
    rho = sim.wall_state()["rho"].copy()
    st = N.stream_ptr()
    N.call("sph_mdbc_wall_density", _ref(sim.fluid_view), _ref(sim.wall_view), N.ptr(sim.grid), _ref(sim.params), st)
    a, d = torch.empty_like(acc), torch.empty_like(dpdt)
    gr = torch.empty(2 * sim.n, device=cuda)
    scr = torch.empty(N.load().sph_deltasph_scratch_bytes(sim.n) // 8 + 1, dtype=torch.int64, device=cuda)
    N.call("sph_deltasph_forces", _ref(sim.fluid_view), _ref(sim.wall_view), N.ptr(sim.grid), _ref(sim.params),
           N.ptr(d), N.ptr(a), None, N.ptr(gr), N.ptr(scr), scr.numel() * 8, st)
    assert torch.equal(a, acc) and torch.equal(d, dpdt)
    assert np.array_equal(sim.wall_state()["rho"], rho)
    t0 = float(sim.time.item())
    sim.step()
    assert float(sim.time.item()) == t0 + float(sim.dt.item())


@pytest.mark.parametrize("n", [1, 255, 257, 5000])
def test_rk_stage(cuda, n):
    from pytorchsph_gb300 import _native as N
    r = lambda *s: torch.randn(s, device=cuda)
    x0, v0, r0 = r(n, 2), r(n, 2), r(n)
    dt, st = torch.full((1,), 1e-3, device=cuda), N.stream_ptr()
    sums = [[torch.zeros_like(t) for t in (x0, v0, r0)] for _ in range(2)]
    status = torch.zeros(1, dtype=torch.int32, device=cuda)
    time = torch.full((1,), 2.5, dtype=torch.float64, device=cuda)
    for k, (c, w) in enumerate([(0.5, 1.0), (0.5, 2.0), (1.0, 2.0), (1.0 / 6.0, 1.0)]):
        rates = [r(n, 2), r(n, 2), r(n)]
        out = [[torch.empty_like(t) for t in (x0, v0, r0)] for _ in range(2)]
        p = lambda ts: [N.ptr(t) for t in ts]
        N.call("sph_rk_accumulate", n, *p(rates), w, int(k == 0), *p(sums[0]), st)
        N.call("sph_rk_axpy", n, *p((x0, v0, r0)), *p(rates if k < 3 else sums[0]), N.ptr(dt), c, 1000.0, *p(out[0]),
               N.ptr(status), st)
        N.call("sph_rk_stage", n, *p((x0, v0, r0)), *p(rates), w, int(k == 0), int(k == 3), *p(sums[1]), N.ptr(dt), c,
               1000.0, *p(out[1]), N.ptr(status), N.ptr(time) if k == 3 else None, st)
        for a, b in zip(sums[0] + out[0], sums[1] + out[1]):
            assert torch.equal(a, b)
    assert float(time.item()) == 2.5 + float(np.float32(1e-3)) and int(status.item()) == 0
