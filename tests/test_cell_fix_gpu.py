"""The counting sort's order inside cells, with the rows it moves, at cell sizes around its
limits (48 per thread rank, 1024 per block rank, 2048 per block sort) and with large cells
that begin anywhere in a block, against numpy's stable sort: integers and copies, equal."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[1], [48, 49, 48, 50], [49] * 23, [255, 1, 256, 257], [3, 1024, 1025, 7],
                                   [2048, 5, 2048], [100] * 40 + [1] * 300 + [2000],
                                   [49] * 3000 + [1025, 2048] + [2] * 60000])   # past 2^18: large cells in a launch
@pytest.mark.parametrize("with_tie", [False, True])
def test_order(cuda, sizes, with_tie):
    from pytorchsph_gb300 import _native as N
    rng = np.random.default_rng(len(sizes))
    cap = len(sizes) + 3
    keys = np.repeat(np.arange(len(sizes)) + 1, sizes).astype(np.int32)
    keys = np.concatenate([keys, np.full(5, cap, np.int32)])        # five outside every cell
    rng.shuffle(keys)
    n = len(keys)
    tie = rng.permutation(n).astype(np.int32) if with_tie else None
    t = lambda a: torch.from_numpy(a).to(cuda)
    i32 = lambda m: torch.empty(m, dtype=torch.int32, device=cuda)
    count = torch.from_numpy(np.bincount(keys, minlength=cap + 1).astype(np.int32)).to(cuda)
    start, order, skeys, status = i32(cap + 2), i32(n), i32(n), torch.zeros(1, dtype=torch.int32, device=cuda)
    rows = [torch.randn(s, device=cuda) for s in ((n,), (n, 2), (n, 4), (n,), (n, 2))]   # past one group of four
    out = [torch.empty_like(r) for r in rows]
    k, eb, ins, outs = N.array_set(list(zip(rows, out)))
    size = N.load().sph_counting_sort_scratch_bytes(n, cap)
    scratch = torch.empty((size + 7) // 8, dtype=torch.int64, device=cuda)
    dk, dt = t(keys), t(tie) if with_tie else None
    N.call("sph_counting_sort_permute", N.ptr(dk), n, cap, N.ptr(count), N.ptr(start), N.ptr(dt), N.ptr(order),
           N.ptr(skeys), k, eb, ins, outs, N.ptr(status), N.ptr(scratch), scratch.numel() * 8, N.stream_ptr())
    want = np.lexsort((np.arange(n) if tie is None else tie, keys))
    got = order.cpu().numpy()
    assert int(status.item()) == 0 and np.array_equal(skeys.cpu().numpy(), keys[want])
    inside = n - 5
    assert np.array_equal(got[:inside], want[:inside]) and sorted(got[inside:]) == sorted(want[inside:])
    for r, o in zip(rows, out):
        assert torch.equal(o, r[order.long()])
