"""The extension's per-point query (lanes per point: the reference's visiting order) and the
(i, j)-ordered rows of constructNeighborhoodsCUDA, against all pairs in float32 on the host
and against the per-cell search.  Pair sets and orders are integers: equal."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,spread", [(1, 1.0), (3, 0.2), (33, 0.4), (70, 0.05), (257, 1.0), (700, 0.3)])
@pytest.mark.parametrize("radius,length", [(1, -1), (0, -1), (2, -1), (1, 7)])
def test_rows(cuda, n, spread, radius, length):
    from pytorchsph_gb300 import neighborhoods as NH, neighborSearch as NS
    rng = np.random.default_rng(n)
    x = rng.uniform(0, spread, (n, 2)).astype(np.float32)
    h = rng.uniform(0.06, 0.1, n).astype(np.float32)
    pos, sup = torch.from_numpy(x).cuda(), torch.from_numpy(h).cuda()
    i, j, _, _, state, table, cells = NH.constructNeighborhoodsCUDA(pos, sup, length, searchRadius=radius)
    qMin, hMax, order, sp, ss = state
    ci, cum, span, cells_x = cells
    assert i.dtype == j.dtype == torch.int64
    key = (i * n + j).cpu().numpy()
    assert np.all(np.diff(key) > 0)                          # distinct, in (i, j) order
    rows, cols, *_ = NH.constructNeighborhoods(pos, sup, length, searchRadius=radius)
    assert np.array_equal(np.sort((rows * n + cols).cpu().numpy()), key)
    a, b = NS.buildNeighborListCUDA(pos, sup, sp, ss, table[0], ci, cum, span, order, qMin, hMax, cells_x, table[1],
                                    radius)
    a, b = a.cpu().numpy().astype(np.int64), b.cpu().numpy().astype(np.int64)
    cell = np.ceil((x - qMin.cpu().numpy()) / np.float32(hMax)).astype(np.int64)   # neighborSearch.py:46
    place = np.empty(n, np.int64)
    place[order.cpu().numpy()] = np.arange(n)
    visit = np.lexsort((place[b], cell[b, 1], cell[b, 0], a))   # by row, then cell x, cell y, sorted place
    assert np.array_equal(visit, np.arange(len(a)))
    assert np.array_equal(np.sort(a * n + b), key)
    if radius >= 1:
        d = x[:, None] - x[None]
        near = np.sqrt(d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]) < h[:, None]
        assert np.array_equal(np.flatnonzero(near.ravel()), key)
