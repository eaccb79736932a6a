"""A drop rollout's own neighbor lists and steps (lanes per row, rows past a capacity run
again, rows ordered in a block or from a second array), against the step on the reference's
(i, j)-ordered lists and, for the adjoint, against autograd through a dense float64
restatement of the step.

Tolerances.  float32 rows are summed in the same order by both, so states are equal.  float64
rows are summed in another order: a step moves x by dt^2 a, whose terms are below 1e-2 of
the spacing, so 60 terms differ by less than 60 * 1.1e-16 of it; 1e-12 of the extent is
held.  The adjoint's derivatives are algebraically those of the dense step: 1e-10 of the
largest component in float64.  In float32 the derivative of a step's velocity is
dt^2 d a / dx, of order (0.1)^2 per pair, and its entries carry the rounding of x_i - x_j (|x| / h
< 6 times 6e-8) and of some 30 operations: about 2e-6 * 0.01 * 60 pairs * 3 steps; 1e-4
of the largest component is held."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
STEPS, C0 = 3, 10.0


def blob(n, seed):
    """n particles on a jittered lattice (spacing 0.05, support 0.15) with random velocities."""
    rng = np.random.default_rng(seed)
    m = int(np.ceil(np.sqrt(n)))
    g = np.stack(np.meshgrid(np.arange(m), np.arange(m), indexing="ij"), -1).reshape(-1, 2)[:n]
    pos = ((g - 0.5 * m) * 0.05 + rng.uniform(-0.008, 0.008, (n, 2))).astype(np.float32)
    f = lambda a: np.asarray(a, np.float32)
    ext = 0.05 * m + 0.5
    return {"pos": pos, "vel": f(rng.uniform(-0.5, 0.5, (n, 2))), "rho": f(rng.uniform(0.99, 1.01, n)),
            "area": f(np.full(n, 0.0025)), "support": f(np.full(n, 0.15)), "h": float(np.float32(0.15)),
            "vmin": f([-ext, -ext]), "vmax": f([ext, ext])}


def dense_rollout(sc, v, alpha, dt, steps):
    """The step of src/deltaSPH.py:146-200 (point source, MOG, nu 0.001, delta 0.1) over all pairs."""
    t = lambda a: torch.from_numpy(np.asarray(a, np.float64))
    x, rt, A, h, rho0 = t(sc["pos"]), t(sc["rho"]), t(sc["area"]), sc["h"], 1000.0
    eye = torch.eye(len(x), dtype=torch.bool)
    for _ in range(steps):
        d, w = x[:, None] - x[None], v[:, None] - v[None]
        r2 = (d * d).sum(-1)
        near = ~eye & (r2.detach() < h * h)
        r = torch.sqrt(torch.where(near, r2, torch.ones_like(r2)))
        gd = torch.where(near, -(20 * 7 / (np.pi * h ** 4)) * (1 - r / h) ** 3, torch.zeros_like(r))
        rho, p = rho0 * rt, rho0 * C0 * C0 / 7 * (rt ** 7 - 1)
        V, R2, s = (A / rt)[None], r2 + 0.1 * h * h, (w * d).sum(-1)
        rj, rs = rho[None], rho[:, None] + rho[None]
        k = -(p[:, None] + p[None]) * V / rho[:, None] * gd + alpha * h * C0 * torch.clamp(s, max=0) / R2 * V * rj / rs * gd
        lam = 8 * rj * V * rho[:, None] * 0.001 * r2 * gd / (rs * rs * R2)
        a = (k[..., None] * d).sum(1) + (lam[..., None] * w).sum(1) - x
        dp = (s * gd * V * rj).sum(1) - (0.1 * h * C0 * 2 * (rj - rho[:, None]) / R2 * r2 * gd * V).sum(1)
        v, x, rt = v + dt * a, x + dt * (v + dt * a), rt + dt * dp / rho0
    return x


@pytest.mark.parametrize("n", [1, 2, 7, 9, 33, 130])
@pytest.mark.parametrize("fp64", [True, False])
@pytest.mark.parametrize("capacity", [None, 1, 600])
def test_rollout_and_adjoint(cuda, n, fp64, capacity):
    from pytorchsph_gb300.adjoint import DropRollout
    sc = blob(n, n)
    dt = 0.1 * sc["h"] / C0
    r = DropRollout(sc, C0, dt, fp64=fp64, checkpoint_every=2, device=cuda)
    if capacity:
        r._row_cap = capacity
    v0 = torch.as_tensor(sc["vel"], dtype=r.dtype, device=cuda)
    xT, _ = r.rollout(v0, 0.05, STEPS)
    assert r._row_cap > 1 or n == 1
    x, v, rho = r.x0.clone(), v0.clone(), r.rho0.clone()
    for _ in range(STEPS):
        r.step(x, v, rho, 0.05)
    if fp64:
        assert float((xT - x).abs().max()) <= 1e-12 * float(x.abs().max())
    else:
        assert torch.equal(xT, x)

    target = torch.from_numpy(sc["pos"].astype(np.float64) + 0.01)
    vd = torch.from_numpy(sc["vel"].astype(np.float64)).requires_grad_()
    al = torch.tensor(0.05, dtype=torch.float64, requires_grad=True)
    loss = ((dense_rollout(sc, vd, al, dt, STEPS) - target) ** 2).sum() / n
    gv, ga = torch.autograd.grad(loss, [vd, al])
    got, gvr, gar = r.loss_and_grad(v0, 0.05, target.to(cuda), STEPS)
    tol = 1e-10 if fp64 else 1e-4
    gvr = torch.as_tensor(gvr).double().cpu().reshape(n, 2)
    assert float((gvr - gv).abs().max()) <= tol * float(gv.abs().max())
    assert abs(got - loss.item()) <= tol * loss.item()
    if fp64:
        assert abs(float(gar) - float(ga)) <= 1e-8 * max(abs(float(ga)), 1e-30) + 1e-24


def test_out_of_domain_is_refused(cuda):
    from pytorchsph_gb300 import _native as N
    from pytorchsph_gb300.adjoint import DropRollout
    sc = blob(33, 3)
    r = DropRollout(sc, C0, 0.5, fp64=True, device=cuda)
    v0 = torch.full((33, 2), 50.0, dtype=torch.float64, device=cuda)
    with pytest.raises(N.SPHError):
        r.rollout(v0, 0.0, 3)
    r.rollout(torch.zeros_like(v0), 0.0, 0)
    assert r.rollout(v0 * 1e-3, 0.0, 1)[0].shape == (33, 2)


@pytest.mark.parametrize("n", [2432, 2433, 12288, 12289])
@pytest.mark.parametrize("fp64", [True, False])
def test_lanes_by_size(cuda, n, fp64):
    """Sizes on both sides of the lanes' limits: the rollout against the (i, j)-ordered step (the same
    bits in float32), and the gradient of the sum of positions, which one step at rest moves
    as dt to each component (pressure and viscosity are pair forces of equal masses: they
    sum to zero within 30 roundings of dt^2 a, below 1e-5 of dt; gravity's point source
    takes dt^2 off)."""
    from pytorchsph_gb300.adjoint import DropRollout
    sc = blob(n, n)
    dt = 0.1 * sc["h"] / C0
    r = DropRollout(sc, C0, dt, fp64=fp64, device=cuda)
    v0 = torch.as_tensor(sc["vel"], dtype=r.dtype, device=cuda)
    xT, _ = r.rollout(v0, 0.05, 2)
    x, v, rho = r.x0.clone(), v0.clone(), r.rho0.clone()
    for _ in range(2):
        r.step(x, v, rho, 0.05)
    assert torch.equal(xT, x) if not fp64 else float((xT - x).abs().max()) <= 1e-12 * float(x.abs().max())
    (_, *_), _, record = r._forward(v0, 0.05, 1, record=True)
    gv, _ = r._backward(record, 0.05, 1, torch.ones((n, 2), dtype=r.dtype, device=cuda))
    assert float((gv.mean(0) - dt).abs().max()) <= 1e-3 * dt
