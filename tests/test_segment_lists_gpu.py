"""A particle's segment list holds its non-empty segments, whatever the size of the launch: small
launches (four lanes per particle) against large ones (one), at supports whose cell rows have
segments without a neighbor.  Lists are integers, and a scene's state does not depend on what
is stepped beside it: equal."""
import ctypes
import dataclasses

import numpy as np
import pytest
import torch

import test_serve_gpu as serve

pytestmark = pytest.mark.gpu


def block(nx, ratio, walls):
    """A jittered block of nx x nx particles, support `ratio` spacings, in a domain with room beside it."""
    from pytorchsph_gb300 import workloads
    dx = 0.01
    sc = workloads.dam_break(nx, nx, dx, (2 * nx * dx, 2 * nx * dx), layers=int(np.ceil(ratio)) if walls else 1)
    rng = np.random.default_rng(nx)
    n, h = len(sc["pos"]), np.float32(ratio * dx)
    sc["pos"] = (sc["pos"] + rng.uniform(-0.1 * dx, 0.1 * dx, (n, 2))).astype(np.float32)
    sc["vel"] = rng.uniform(-0.1, 0.1, (n, 2)).astype(np.float32)
    if not walls:
        sc.update({k: sc[k][:0] for k in ("wall_pos", "ghost_pos", "wall_area")})
    sc.update(support=np.full(n, h, np.float32), h=float(h), vmin=np.full(2, -2 * h, np.float32),
              vmax=np.full(2, 4 * nx * dx + 6, np.float32))
    return sc


def segment_counts(sim, n):
    """Segment counts of the particles 0 .. n - 1 (-1: more than a list holds) of the last right-hand side."""
    from pytorchsph_gb300 import _native as N
    at = [ctypes.c_size_t() for _ in range(3)]
    most = ctypes.c_int32()
    N.call("sph_deltasph_segment_lists", sim.n, *map(ctypes.byref, at), ctypes.byref(most))
    scr = sim.ws.bytes("forces_scratch", N.load().sph_deltasph_scratch_bytes(sim.n)).view(torch.uint8)
    first = -scr.data_ptr() % 32 + at[2].value
    counts = scr[first:first + 4 * sim.n].view(torch.int32)
    out = torch.empty_like(counts)
    out[sim.arr["uid"].long()] = counts
    return out[:n]


@pytest.mark.parametrize("ratio", [2.0, 3.0, 3.7, 4.0, 4.5, 5.0, 6.0])
@pytest.mark.parametrize("walls", [True, False])
def test_counts_do_not_depend_on_the_launch(cuda, ratio, walls):
    from pytorchsph_gb300.sim import SimConfig, Simulation
    small = block(60, ratio, walls)
    n, more = 3600, 32768
    far = np.stack(np.meshgrid(np.arange(256), np.arange(128)), -1).reshape(-1, 2) * 0.01 + 4.0
    large = dict(small, pos=np.concatenate([small["pos"], far.astype(np.float32)]))
    for k, v in (("vel", np.zeros((more, 2))), ("rho", np.ones(more)), ("area", np.full(more, 1e-4)),
                 ("support", np.full(more, small["support"][0]))):
        large[k] = np.concatenate([small[k], v.astype(np.float32)])
    counts = []
    for sc in (small, large):
        sim = Simulation(sc, SimConfig(dt=1e-5, c0=10.0, density_diffusion="deltaSPH"), cuda, pairs="cells")
        sim.rhs()
        assert int(sim.status.item()) == 0
        counts.append(segment_counts(sim, n).clone())
    assert torch.equal(*counts)
    if ratio <= 4.5:
        assert int(counts[0].min()) > 0


@pytest.mark.parametrize("tpp", [1, 2, 4])
@pytest.mark.parametrize("ratio", [4.0, 5.0])
def test_a_scene_steps_alike_in_any_mix(cuda, tpp, ratio):
    from pytorchsph_gb300.serve import SceneSpec
    from pytorchsph_gb300.sim import SimConfig
    cfg = SimConfig(dt=1e-5, c0=10.0, density_diffusion="deltaSPH")
    A, B = (serve.configured(SceneSpec(block(nx, ratio, True), cfg), 1, tpp) for nx in (60, 190))
    alone = serve.run_batch([A], 3, cuda)[0]
    beside = serve.run_batch([A, B], 3, cuda)[0]
    assert serve.same(alone, beside)
