"""Query pairs by lanes (searchExisting's outputs from the fill) and the grouping of pairs by
column, at point counts and row lengths around the lanes.  Pairs are integers: equal to all
pairs in the reference's predicate, in the order of the plain query; the geometry is the
same float32 expression (a product may be fused): 4 units in the last place."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [0, 1, 4, 5, 130])
@pytest.mark.parametrize("ratio,radius", [(1, 1), (1, 0), (1, 2), (2, 1)])
def test_query_pairs(cuda, m, ratio, radius):
    from pytorchsph_gb300.search import GridSearch
    rng = np.random.default_rng(m)
    n = 700
    x = rng.uniform(0, 1, (n, 2)).astype(np.float32)
    q = rng.uniform(-0.3, 1.3, (m, 2)).astype(np.float32)     # some outside the grid
    hq = rng.uniform(0.04, 0.1, m).astype(np.float32)
    t = lambda a: torch.from_numpy(a).to(cuda)
    res = GridSearch(cuda, cell_ratio=ratio).run(t(x), torch.full((n,), 0.1, device=cuda), density=False)
    rows, cols = res.query(t(q), t(hq), radius)
    pairs, dist, radial, off = res.query_pairs(t(q), t(hq), t(x), 1e-7, radius)
    assert torch.equal(pairs[0], rows.long()) and torch.equal(pairs[1], cols.long())
    r, c = pairs.cpu().numpy()
    assert np.array_equal(off.cpu().numpy(), np.searchsorted(r, np.arange(m + 1)))
    if radius >= 1:
        d = q[:, None] - x[None]
        near = np.sqrt(d[..., 0] ** 2 + d[..., 1] ** 2) < hq[:, None]
        assert np.array_equal(np.sort(r * n + c), np.flatnonzero(near.ravel()))
    d = q[r].astype(np.float64) - x[c]
    length = np.linalg.norm(d, axis=1)
    np.testing.assert_allclose(radial.cpu().numpy(), length / hq[r], rtol=4 * 6e-8)
    np.testing.assert_allclose(dist.cpu().numpy(), d / length[:, None], rtol=4 * 6e-8 + 1e-7, atol=1e-7)


@pytest.mark.parametrize("lengths", [[0, 1, 2], [8, 9, 0, 7], [31, 32, 33, 1], [40, 3, 64, 0, 0, 5], [1] * 33])
def test_pairs_by_column(cuda, lengths):
    from pytorchsph_gb300 import modules
    rng = np.random.default_rng(len(lengths))
    cols = np.repeat(np.arange(len(lengths)), lengths)
    rng.shuffle(cols)
    rows = np.sort(rng.integers(0, 9, len(cols)))
    P, n = len(cols), len(lengths)
    nb = torch.from_numpy(np.stack([rows, cols])).to(cuda)
    w = modules._WallPairs(nb, torch.zeros((P, 2), device=cuda), torch.zeros(P, device=cuda), 9, n)
    assert np.array_equal(w.woff.cpu().numpy(), np.searchsorted(rows, np.arange(10)))
    assert np.array_equal(w.foff.cpu().numpy(), np.concatenate([[0], np.cumsum(lengths)]))
    assert np.array_equal(w.fpairs[:P].cpu().numpy(), np.argsort(cols, kind="stable"))
