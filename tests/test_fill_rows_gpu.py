"""The CSR fill from stored segments (rows staged per lane, stored row by row) against the fill
that tests every candidate again: the same columns in the same order, at row lengths around
the stage (48) and the store (32), several segments per row, dense rows (more than 24
segments) among short ones, and column buffers that hold only some of the rows."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def search(pos, sup, segments, ratio=1, **kw):
    from pytorchsph_gb300.search import GridSearch
    return GridSearch(pos.device, segments=segments, cell_ratio=ratio).run(pos, sup, density=False, **kw)


@pytest.mark.parametrize("n", [1, 31, 33, 128, 129, 1000])
@pytest.mark.parametrize("row", [1, 31, 33, 47, 49, 97, 400])
@pytest.mark.parametrize("ratio", [1, 2])
def test_rows(cuda, n, row, ratio):
    """About `row` neighbors: n particles in a square whose support circle holds that many."""
    rng = np.random.default_rng(n * row)
    side = np.sqrt(np.pi * max(n, 1) / row) * 0.1   # support 0.1
    x = rng.uniform(0, max(side, 0.02), (n, 2)).astype(np.float32)
    if n == 1000 and row == 97:
        x[:900] = x[:900] * 0.01 + 0.05             # a cluster of dense rows
    pos, sup = torch.from_numpy(x).cuda(), torch.full((n,), 0.1, device=cuda)
    a, b = search(pos, sup, True, ratio), search(pos, sup, False, ratio)
    P = a.num_pairs
    assert torch.equal(a.offsets, b.offsets) and torch.equal(a.cols[:P], b.cols[:P])
    # a buffer that ends inside the list: what fits is the same, and the search is flagged
    for cap in sorted({max(P // 2, 1), P - 1} - {0, P}):
        c = search(pos, sup, True, ratio, pair_capacity=cap, cell_capacity=a.cell_capacity, sync=False)
        fits = int((a.offsets[1:] <= cap).sum())
        end = int(a.offsets[fits])
        assert torch.equal(c.cols[:end], a.cols[:end])
        with pytest.raises(RuntimeError):
            c.check()
