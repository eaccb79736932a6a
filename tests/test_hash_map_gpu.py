"""The hash map by counting and by the radix sort, at table lengths on both sides of the rule
between them (a quarter of the particles, sixteen times them), against numpy: buckets in
order, cells increasing inside a bucket, all integers equal."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 33, 400, 5000, 20000])
@pytest.mark.parametrize("length", ["1", "7", "quarter-", "quarter", "n", "16n", "16n+"])
def test_hash_map(cuda, n, length):
    from pytorchsph_gb300 import neighborhoods as NH
    L = {"1": 1, "7": 7, "quarter-": max(n // 4 - 1, 1), "quarter": max(n // 4, 1), "n": n + 3, "16n": 16 * n,
         "16n+": 16 * n + 1}[length]
    rng = np.random.default_rng(n)
    cx = 61
    keys = np.sort(rng.integers(0, cx * 70, n)).astype(np.int32)
    table, ci, cum, span = (t.cpu().numpy() for t in NH.constructHashMap(
        None, None, torch.from_numpy(keys).to(cuda), None, L, cx))
    cells, first, count = np.unique(keys, return_index=True, return_counts=True)
    h = (cells.astype(np.int64) % cx * 3 + cells.astype(np.int64) // cx * 5) % L
    by = np.lexsort((cells, h))
    assert np.array_equal(ci, cells[by]) and np.array_equal(cum, count[by]) and np.array_equal(span, first[by])
    per = np.bincount(h, minlength=L)
    begin = np.concatenate([[0], np.cumsum(per)[:-1]])
    assert np.array_equal(table[:, 1], per)
    assert np.array_equal(table[:, 0], np.where(per > 0, begin, -1))
