"""(i, j)-ordered pair rows at the lengths where a warp's tile of 32 columns begins, ends and
repeats: clusters of m particles within one support of each other give rows of exactly m
columns, checked against a host sort of the CSR search's own pairs (indices equal; distances
are the float32 formula's, within 2 ulp)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 2, 31, 32, 33, 64, 65, 300])
def test_coo_rows_of_length_m(cuda, m):
    from pytorchsph_gb300.search import GridSearch
    rng = np.random.default_rng(m)
    h = np.float32(0.1)
    centres = np.stack(np.meshgrid([0.25, 1.25, 2.25], [0.25, 1.25]), -1).reshape(-1, 2)
    pos = np.concatenate([c + rng.uniform(-0.03, 0.03, (m, 2)) for c in centres]).astype(np.float32)
    pos = pos[rng.permutation(len(pos))]
    n = len(pos)
    x = torch.from_numpy(pos).to(cuda)
    res = GridSearch(cuda).run(x, torch.full((n,), float(h), device=cuda), kernel_support=float(h), density=False)
    assert torch.equal(res.counts[:n], torch.full((n,), m, dtype=torch.int32, device=cuda))
    order = res.order[:n].cpu().numpy().astype(np.int64)
    rows = np.repeat(order, m)
    cols = order[res.cols[:n * m].cpu().numpy()]
    want = np.lexsort((cols, rows))
    pairs, dist, radial = res.to_coo()
    assert np.array_equal(pairs.cpu().numpy(), np.stack([rows[want], cols[want]]))
    d = pos[rows[want]] - pos[cols[want]]
    r = np.sqrt((d.astype(np.float64) ** 2).sum(1))
    e = np.where(r[:, None] < 1e-7, 0.0, d / np.where(r, r, 1.0)[:, None])
    ulp = 2.0 ** -23
    assert np.abs(dist.cpu().numpy() - e).max() <= 2 * ulp
    assert np.abs(radial.cpu().numpy() - r / float(h)).max() <= 2 * ulp
    assert res.to_coo(distances=False)[1] is None
