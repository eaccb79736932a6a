"""The CSR fill at its own limits: a warp's 32 rows are built in a stage of 1,280 columns (rows of 40
in one pass, of 41 in two, .. of more than 640 one by one), and the span is stored in 16-byte
pieces from wherever it begins.  Clusters of m particles give rows of m columns; against the
fill that tests every candidate again: integers, equal."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [20, 39, 40, 41, 80, 81, 160, 161, 320, 321, 639, 640, 641, 700])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_spans(cuda, m, shift):
    from pytorchsph_gb300.search import GridSearch
    rng = np.random.default_rng(m)
    few = max(3, 200 // m + 1)
    # `shift` lone particles come first in cell order and move every span by as many columns
    pos = [np.stack([np.arange(shift) + 0.05, np.full(shift, 0.05)], 1)]
    pos += [[5.0 + k, 3.0] + rng.uniform(0, 0.05, (m, 2)) for k in range(few)]
    pos.append(np.stack([np.arange(40) * 0.15 + 1, np.full(40, 6.0)], 1))   # short rows in the last warps
    x = torch.from_numpy(np.concatenate(pos).astype(np.float32)).to(cuda)
    sup = torch.full((len(x),), 0.1, device=cuda)
    a, b = (GridSearch(cuda, segments=s).run(x, sup, density=False) for s in (True, False))
    P = a.num_pairs
    assert P == shift + few * m * m + 40
    assert torch.equal(a.offsets, b.offsets) and torch.equal(a.cols[:P], b.cols[:P])
