"""The search grid at particle counts around the one-block limit and its loop, against numpy in
float32 (src/modules/neighborSearch.py:34-46): equal, with and without a given domain, and flagged
for one non-finite value anywhere."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 1025, 8191, 8192, 8193, 200000])
@pytest.mark.parametrize("domain", [False, True])
def test_grid(cuda, n, domain):
    from pytorchsph_gb300 import _native as N
    from pytorchsph_gb300.search import GridSearch, grid_from_bytes
    rng = np.random.default_rng(n)
    f = np.float32
    x = rng.uniform(-3, 5, (n, 2)).astype(f)
    h = rng.uniform(0.05, 0.1, n).astype(f)
    lo, hi = (np.array([-4, -4], f), np.array([6, 6], f)) if domain else (None, None)
    s = GridSearch(cuda)
    g = grid_from_bytes(s.grid(torch.from_numpy(x).cuda(), torch.from_numpy(h).cuda(), lo, hi))
    hm = h.max()
    qmin = (lo if domain else x.min(0)) - hm
    qmax = (hi if domain else x.max(0)) + f(2) * hm
    cells = np.ceil((qmax - qmin) / hm).astype(int)
    assert g["qmin"] == (qmin[0], qmin[1]) and g["hmax"] == hm
    assert (g["cells_x"], g["cells_y"], g["num_cells"]) == (cells[0], cells[1], cells[0] * cells[1])
    for k in {0, n // 2, n - 1}:
        y = x.copy()
        y[k, 1] = np.inf
        with pytest.raises(N.SPHError):
            s.auto_cell_capacity(torch.from_numpy(y).cuda(), torch.from_numpy(h).cuda(), lo, hi)
