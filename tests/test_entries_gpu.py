"""C entries that this package itself no longer calls, against those it does: the adjoint of a step over
int64 lists, and the geometry of query pairs.  The same operations in the same order: equal."""
import ctypes

import numpy as np
import pytest
import torch

import test_drop_lists_gpu as drops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 2433, 9729])
@pytest.mark.parametrize("fp64", [True, False])
def test_drop_adjoint(cuda, n, fp64):
    from pytorchsph_gb300 import _native as N
    from pytorchsph_gb300.adjoint import DropRollout
    sc = drops.blob(n, n)
    r = DropRollout(sc, drops.C0, 0.1 * sc["h"] / drops.C0, fp64=fp64, device=cuda)
    r.P.alpha = 0.05
    off, cols = r.pairs(r.x0)
    new = lambda *s: torch.randn(*s, dtype=r.dtype, device=cuda)
    v, lx, lv, lr = torch.as_tensor(sc["vel"], dtype=r.dtype, device=cuda), new(n, 2), new(n, 2), new(n)
    got = []
    for name, c, room in (("sph_drop_adjoint", cols, []), ("sph_drop_adjoint_step", cols.to(torch.int32), [0])):
        out = [torch.empty_like(t) for t in (lx, lv, lr)] + [torch.zeros_like(lr)]
        N.call(name, int(fp64), n, N.ptr(off), N.ptr(c), *room, N.ptr(r.x0), N.ptr(v), N.ptr(r.rho0), N.ptr(r.area),
               ctypes.byref(r.P), r.dt, N.ptr(lx), N.ptr(lv), N.ptr(lr), *map(N.ptr, out), N.stream_ptr())
        if room:   # adds to dalpha
            once = out[3].clone()
            N.call(name, int(fp64), n, N.ptr(off), N.ptr(c), *room, N.ptr(r.x0), N.ptr(v), N.ptr(r.rho0),
                   N.ptr(r.area), ctypes.byref(r.P), r.dt, N.ptr(lx), N.ptr(lv), N.ptr(lr), *map(N.ptr, out),
                   N.stream_ptr())
            assert torch.equal(out[3], once + once)
            out[3] = once
        got.append(out)
    assert all(torch.equal(a, b) for a, b in zip(*got))


def test_pair_geometry(cuda):
    from pytorchsph_gb300 import _native as N
    from pytorchsph_gb300.search import GridSearch
    rng = np.random.default_rng(1)
    t = lambda a: torch.from_numpy(a.astype(np.float32)).to(cuda)
    x, q = t(rng.uniform(0, 1, (700, 2))), t(rng.uniform(-0.2, 1.2, (300, 2)))
    q[::7] = x[:43]   # distance 0
    hq = t(rng.uniform(0.02, 0.1, 300))
    s = GridSearch(cuda).run(x, torch.full((700,), 0.1, device=cuda), density=False)
    pairs, dist, radial, rows = s.query_pairs(q, hq, x, 1e-7)
    r, c = s.query(q, hq)
    d, g = torch.empty_like(dist), torch.empty_like(radial)
    N.call("sph_pair_geometry", N.ptr(r), N.ptr(c), len(r), N.ptr(q), N.ptr(x), N.ptr(hq), 1e-7, N.ptr(d), N.ptr(g),
           N.stream_ptr())
    assert len(r) > 300 and torch.equal(pairs, torch.stack([r, c]).long())
    assert torch.equal(d, dist) and torch.equal(g, radial)
    assert torch.equal(rows[1:].long(), torch.bincount(r.long(), minlength=300).cumsum(0)) and int(rows[0]) == 0
