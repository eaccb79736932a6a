"""float32 rollout sums keep the order of their rows: the step, the gradient and each particle's share
of dL/d alpha are the same bits with 4 and with 8 lanes per row, and those of the list in
increasing column order.  The number of lanes follows the number of particles, so a set
is taken alone and with far-away particles beside it that lift the launch past a line."""
import numpy as np
import pytest
import torch

import test_drop_lists_gpu as drops

pytestmark = pytest.mark.gpu


def shares(r, v0, record, steps, grad):
    """(gradient with respect to v0, dL/d alpha per particle) of a record's last step backwards."""
    import ctypes
    from pytorchsph_gb300 import _native as N
    start, mid, counts, cols, cap = record
    n = r.n
    cur = [grad.clone(), torch.zeros_like(grad), torch.zeros_like(r.rho0)]
    da = torch.zeros(n, dtype=r.dtype, device=r.dev)
    for k in reversed(range(steps)):
        state = start if k == 0 else [t[k - 1] for t in mid]
        nxt = [torch.empty_like(t) for t in cur]
        N.call("sph_drop_adjoint_step", int(r.fp64), n, N.ptr(counts[k]), N.ptr(cols[k]), cap, *map(N.ptr, state),
               N.ptr(r.area), ctypes.byref(r.P), r.dt, *map(N.ptr, cur), *map(N.ptr, nxt), N.ptr(da), N.stream_ptr())
        cur = nxt
    return cur[1], da


@pytest.mark.parametrize("far", [9728, 9729, 24320, 24321])
def test_lanes_keep_the_bits(cuda, far):
    """Lines: the adjoint's at 9,728 particles, the right-hand side's at 24,320."""
    from pytorchsph_gb300.adjoint import DropRollout
    n, steps = 600, 2
    sc = drops.blob(n, 5)
    more = drops.blob(far - n, 6)
    more["pos"] = more["pos"] + np.float32(40.0)
    both = {k: np.concatenate([sc[k], more[k]]) if k in ("pos", "vel", "rho", "area", "support") else sc[k] for k in sc}
    dt = 0.1 * sc["h"] / drops.C0
    got = []
    for scene, size in ((sc, n), (both, far)):
        scene = dict(scene, vmin=np.float32([-60, -60]), vmax=np.float32([60, 60]))
        r = DropRollout(scene, drops.C0, dt, fp64=False, device=cuda)
        assert r.n == size
        v0 = torch.as_tensor(scene["vel"], device=cuda)
        end, _, record = r._forward(v0, 0.05, steps, record=True)
        grad = torch.linspace(-1, 1, 2 * n, device=cuda).view(n, 2)
        full = torch.zeros((size, 2), device=cuda)
        full[:n] = grad
        gv, da = shares(r, v0, record, steps, full)
        got.append([end[0][:n], end[1][:n], end[2][:n], gv[:n], da[:n]])
        x, v, rho = r.x0.clone(), v0.clone(), r.rho0.clone()
        for _ in range(steps):
            r.step(x, v, rho, 0.05)
        assert torch.equal(x, end[0]) and torch.equal(v, end[1]) and torch.equal(rho, end[2])
    for a, b in zip(*got):
        assert torch.equal(a, b)
    assert float(got[0][4].abs().max()) > 0


def test_alpha_gradient_in_float(cuda):
    """dL/d alpha of a float32 rollout against autograd through the dense float64 step.  A particle's
    share is a sum of ~30 float32 terms of both signs, the total a sum over particles of shares
    of both signs: each share is off by at most 60 roundings of its largest terms, so the
    total by 60 * 6e-8 of the sum of the shares' magnitudes times the cancellation inside a
    share, at most its 30 terms; 60 * 30 * 6e-8 = 1.1e-4 of that sum is held, times the steps."""
    from pytorchsph_gb300.adjoint import DropRollout
    n, steps = 600, 3
    sc = drops.blob(n, 9)
    dt = 0.1 * sc["h"] / drops.C0
    r = DropRollout(sc, drops.C0, dt, fp64=False, device=cuda)
    target = torch.from_numpy(sc["pos"].astype(np.float64) + 0.01)
    vd = torch.from_numpy(sc["vel"].astype(np.float64))
    al = torch.tensor(0.05, dtype=torch.float64, requires_grad=True)
    ((drops.dense_rollout(sc, vd, al, dt, steps) - target) ** 2).sum().div(n).backward()
    v0 = torch.as_tensor(sc["vel"], device=cuda)
    end, _, record = r._forward(v0, 0.05, steps, record=True)
    _, da = shares(r, v0, record, steps, (2.0 / n) * (end[0] - target.to(cuda).float()))
    _, _, ga = r.loss_and_grad(v0, 0.05, target.to(cuda), steps)
    assert abs(float(ga) - float(al.grad)) <= 1.1e-4 * steps * float(da.double().abs().sum())
    assert float(ga) == float(da.sum())
