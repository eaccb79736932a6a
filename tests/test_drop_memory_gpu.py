"""Drop rollouts whose particles gather in one place: the record's memory follows the rows' lengths, not
the longest row, and states and gradients are those of the slots that hold every row."""
import numpy as np
import pytest
import torch

import test_drop_lists_gpu as drops

pytestmark = pytest.mark.gpu


def gathered(n, clump):
    """A blob of n particles with `clump` more within a support of each other beside it."""
    sc = drops.blob(n, 3)
    rng = np.random.default_rng(clump)
    more = drops.blob(clump, 4)
    more["pos"] = (sc["pos"].max(0) + 0.3 + rng.uniform(0, 0.1, (clump, 2))).astype(np.float32)
    both = {k: np.concatenate([sc[k], more[k]]) if k in ("pos", "vel", "rho", "area", "support") else sc[k] for k in sc}
    ext = np.abs(both["pos"]).max() + 1
    return dict(both, vmin=np.float32([-ext, -ext]), vmax=np.float32([ext, ext]))


@pytest.mark.parametrize("fp64", [True, False])
def test_memory_follows_the_rows(cuda, fp64):
    """4,096 particles with rows of 29 and 800 of 800, 30 steps.  Exact int64 lists of every step, as the
    reference's own pairs are kept, take 30 x 8 bytes a pair; the states, one search and its
    pairs' conversion come on top, below a step's 64 bytes a pair: 1.25 times the lists are held
    (slots for the longest row would take 30 x 1,536 x 4 bytes a particle, 4.7 times them)."""
    from pytorchsph_gb300.adjoint import DropRollout
    sc = gathered(4096, 800)
    steps = 30
    r = DropRollout(sc, drops.C0, 1e-5, fp64=fp64, device=cuda)
    v0 = torch.as_tensor(sc["vel"], dtype=r.dtype, device=cuda)
    pairs = r.pairs(r.x0)[1].numel()
    assert pairs > 800 * 800
    target = r.x0 + 0.01
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    base = torch.cuda.memory_allocated()
    r.loss_and_grad(v0, 0.05, target, steps)
    peak = torch.cuda.max_memory_allocated() - base
    assert peak < 1.25 * steps * 8 * pairs, (peak, pairs)


@pytest.mark.parametrize("fp64", [True, False])
@pytest.mark.parametrize("clump", [40, 90, 200])
def test_gathered_particles(cuda, fp64, clump):
    """Rows that fit the slots, twice the slots, or neither, against slots given for every row."""
    from pytorchsph_gb300.adjoint import DropRollout
    sc = gathered(300, clump)
    got = []
    for slots in (None, 512):
        r = DropRollout(sc, drops.C0, 1e-5, fp64=fp64, checkpoint_every=2, device=cuda)
        if slots:
            r._row_cap = slots
        v0 = torch.as_tensor(sc["vel"], dtype=r.dtype, device=cuda)
        end, ck = r.rollout(v0, 0.05, 5, checkpoints=True)
        loss, gv, ga = r.loss_and_grad(v0, 0.05, r.x0 + 0.01, 5)
        assert sorted(ck) == [0, 2, 4]
        gx, gax = r.vjp(ck, 0.05, 5, (2.0 / r.n) * (end - r.x0 - 0.01))
        got.append([end, gv, ck[4][1], gx, torch.tensor([loss, ga]), gax])
    for a, b in zip(*got):
        if fp64:   # sums in another order
            assert float((a - b).abs().max()) <= 1e-10 * float(b.abs().max())
        else:
            assert torch.equal(a, b)


def test_autograd_over_lists(cuda):
    """DropRolloutFunction through rows no slots hold, with the backward run twice."""
    from pytorchsph_gb300.adjoint import DropRollout, drop_rollout
    sc = gathered(300, 200)
    r = DropRollout(sc, drops.C0, 1e-5, device=cuda)
    v = torch.as_tensor(sc["vel"], dtype=torch.float64, device=cuda).requires_grad_()
    al = torch.tensor(0.05, dtype=torch.float64, device=cuda, requires_grad=True)
    x = drop_rollout(r, v, al, 4)
    target = r.x0 + 0.01
    gx = (2.0 / r.n) * (x.detach() - target)   # as loss_and_grad forms it
    first = torch.autograd.grad(x, [v, al], gx, retain_graph=True)
    second = torch.autograd.grad(x, [v, al], gx)
    want = r.loss_and_grad(v.detach(), 0.05, target, 4)
    assert all(torch.equal(a, b) for a, b in zip(first, second))
    assert torch.equal(first[0], want[1]) and float(first[1]) == want[2]
