"""Sets with many particles in a cell or a row: order and speed.

Order is compared with a stable sort on the host (integers, equal).  Speed is compared with
another call on the same device over the same number of particles or pairs, as a ratio with
at least a factor of 1.5 between the bar and what the calls take."""
import numpy as np
import pytest
import torch

import test_cell_fix_gpu as cells
import test_pair_rows_gpu as rows

pytestmark = pytest.mark.gpu


def time_us(f, runs=5, repeats=10):
    """The shortest of `repeats` means over `runs` calls, on the device."""
    for _ in range(3):
        f()
    best = float("inf")
    for _ in range(repeats):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        for _ in range(runs):
            f()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3 / runs)
    return best


def graph_of(f):
    f()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        f()
    return g.replay


@pytest.mark.parametrize("sizes", [[320, 321, 49], [320] * 9, [512, 513, 320, 1024], [300] * 200 + [7] * 50,
                                   [49, 319, 1, 2048, 64, 1], [512] * 520 + [320] * 30])
@pytest.mark.parametrize("with_tie", [False, True])
def test_cell_order(cuda, sizes, with_tie):
    """Cells around the block's limits: 320 entries ranked with the block's others, then bitonic
    passes with one, two or four pairs a thread."""
    cells.test_order(cuda, sizes, with_tie)


def test_sort_of_large_cells_in_time(cuda):
    """100,000 particles in cells of 1,000 against cells of 9.  The scatter's atomics on 100 words take
    about 16 us more, the ranks about 20; four times the small cells' 19 us is held."""
    from pytorchsph_gb300 import _native as N
    n, took = 100000, {}
    for size in (9, 1000):
        cap = -(-n // size)
        rng = np.random.default_rng(size)
        keys = torch.from_numpy(rng.permutation(np.arange(n) // size).astype(np.int32)).to(cuda)
        full = torch.bincount(keys.long(), minlength=cap + 1).to(torch.int32)
        i32 = lambda m: torch.empty(m, dtype=torch.int32, device=cuda)
        count, start, order, skeys, status = full.clone(), i32(cap + 2), i32(n), i32(n), torch.zeros_like(full[:1])
        scratch = torch.empty(N.load().sph_counting_sort_scratch_bytes(n, cap) // 8 + 1, dtype=torch.int64, device=cuda)

        def sort():
            count.copy_(full)
            N.call("sph_counting_sort", N.ptr(keys), n, cap, N.ptr(count), N.ptr(start), N.ptr(order), N.ptr(skeys),
                   N.ptr(status), N.ptr(scratch), scratch.numel() * 8, N.stream_ptr())
        took[size] = time_us(graph_of(sort))
        assert torch.equal(order.long(), torch.argsort(keys.long(), stable=True))
    assert took[1000] < 4 * took[9], took


def clusters(n, size, seed=0):
    """n particles in clusters of `size` within a support (0.1) of each other, in random order."""
    rng = np.random.default_rng(seed)
    c = np.arange(n) // size
    pos = np.stack([c % 64, c // 64], 1) * 1.0 + rng.uniform(0, 0.05, (n, 2))
    return torch.from_numpy(rng.permutation(pos).astype(np.float32)).cuda()


def test_fill_of_dense_rows_in_time(cuda):
    """8,192 rows of 1,024 columns, all on the dense list: the fill stores 34 MB and repeats the
    count's candidate tests a warp per row (a third of the count's time); twice it is held."""
    from pytorchsph_gb300 import _native as N
    from pytorchsph_gb300.search import GridSearch
    n = 8192
    pos, sup = clusters(n, 1024), torch.full((n,), 0.1, device=cuda)
    s = GridSearch(cuda)
    r = s.run(pos, sup, density=False)
    assert r.num_pairs == n * 1024
    seg = s.ws.bytes("segments", N.load().sph_nl_segments_scratch_bytes(n))
    head = (N.ptr(r.xy), N.ptr(r.sh))
    grid = (n, N.ptr(r.keys), N.ptr(r.cell_start), N.ptr(r.grid), r.cell_capacity, 1)

    def count():
        N.call("sph_nl_count_segments", *head, None, *grid, 0.0, N.ptr(r.counts), None, N.ptr(seg), seg.numel() * 8,
               N.stream_ptr())

    def fill():
        N.call("sph_nl_fill_segments", *head, *grid, N.ptr(r.offsets), r.pair_capacity, N.ptr(r.cols), N.ptr(r.status),
               N.ptr(seg), seg.numel() * 8, N.stream_ptr())
    want = r.cols.clone()
    counted = time_us(graph_of(count))
    r.cols.zero_()
    filled = time_us(graph_of(fill))
    assert torch.equal(r.cols, want) and filled < 2 * counted, (filled, counted)


@pytest.mark.parametrize("m", [111, 112, 113, 255, 256, 257, 511, 513, 1025, 2040])
def test_coo_rows(cuda, m):
    """Rows around the length from which they are sorted, and the sort's pieces of 256."""
    rows.test_coo_rows_of_length_m(cuda, m)


def sorts_of(pairs):
    """Two stable sorts of a pair list, by column and by row (src/modules/neighborSearch.py:153-157)."""
    i, j = (t.to(torch.int32) for t in pairs)
    perm = torch.randperm(len(i), device=i.device)
    i, j = i[perm], j[perm]

    def f():
        b, at = torch.sort(j, stable=True)
        a, at2 = torch.sort(i[at], stable=True)
        return a, b[at2]
    return f


def test_coo_of_long_rows_in_time(cuda):
    """8,192 rows of 2,048 columns against two sorts of the same 16.8 M pairs without their distances."""
    from pytorchsph_gb300.search import GridSearch
    n = 8192
    r = GridSearch(cuda).run(clusters(n, 2048), torch.full((n,), 0.1, device=cuda), kernel_support=0.1, density=False)
    pairs = r.to_coo()[0]
    key = pairs[0] * n + pairs[1]
    assert bool((key[1:] > key[:-1]).all()) and len(key) == n * 2048
    taken, sorts = time_us(lambda: r.to_coo()), time_us(sorts_of(pairs))
    assert taken < sorts, (taken, sorts)


@pytest.mark.parametrize("m", [112, 113, 256, 257, 2049, 5000])
def test_constructed_pairs_of_long_rows(cuda, m):
    """constructNeighborhoodsCUDA with rows of m columns beside rows of one: (i, j) order and equal to all
    pairs (the points of a cluster are within a support of each other)."""
    from pytorchsph_gb300 import neighborhoods
    rng = np.random.default_rng(m)
    x = np.concatenate([rng.uniform(0, 0.05, (m, 2)), np.stack([np.arange(40) + 1.0, np.zeros(40)], 1)])
    perm = rng.permutation(len(x))
    x, inside = x[perm].astype(np.float32), (np.arange(len(x)) < m)[perm]
    i, j, *_ = neighborhoods.constructNeighborhoodsCUDA(torch.from_numpy(x).to(cuda),
                                                        torch.full((len(x),), 0.1, device=cuda))
    c = np.flatnonzero(inside)
    one = np.flatnonzero(~inside)
    rows = np.concatenate([np.repeat(c, m), one])
    cols = np.concatenate([np.tile(c, m), one])
    want = np.lexsort((cols, rows))
    assert np.array_equal(i.cpu().numpy(), rows[want]) and np.array_equal(j.cpu().numpy(), cols[want])


def test_constructed_pairs_of_long_rows_in_time(cuda):
    """8,192 rows of 4,096 columns: the order against two sorts of the 33.6 M pairs."""
    from pytorchsph_gb300 import _native as N, neighborhoods
    n, m = 8192, 4096
    i, j, *_ = neighborhoods.constructNeighborhoodsCUDA(clusters(n, m), torch.full((n,), 0.1, device=cuda))
    assert len(i) == n * m
    off = torch.arange(0, n * m + 1, m, device=cuda)
    cols = j.view(n, m)[:, torch.randperm(m, device=cuda)].to(torch.int32).contiguous()
    a, b = torch.empty_like(i), torch.empty_like(j)
    taken = time_us(lambda: N.call("sph_nl_pairs_in_order", n, N.ptr(off), N.ptr(cols), N.ptr(a), N.ptr(b),
                                   N.stream_ptr()))
    sorts = time_us(sorts_of((i, j)))
    assert torch.equal(a, i) and torch.equal(b, j) and taken < sorts, (taken, sorts)


def test_grids_of_many_small_sets(cuda):
    """256, 257, 4,096 and 4,097 sets of 1 to 9,000 particles, among them lengths around a block's loads,
    against the grid of each set alone (the same words); and 100,000 sets of 10 in time, against
    one grid of all their particles (some 8 us): a block of 256 threads each takes about 18
    times that, 35 times is held."""
    from pytorchsph_gb300 import _native as N
    rng = np.random.default_rng(0)
    i32 = lambda m: torch.zeros(m, dtype=torch.int32, device=cuda)
    for sets in (1, 256, 257, 4096, 4097):
        sizes = rng.integers(1, 40, sets)
        sizes[:7] = [1, 4096, 4097, 9000, 3841, 8191, 8193][:sets]
        off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
        pos = torch.rand(int(off[-1]), 2, device=cuda) * 3
        sup = torch.rand(int(off[-1]), device=cuda) * 0.1 + 0.05
        grids, one, status = i32(8 * sets), i32(8), i32(1)
        seg = torch.from_numpy(off).to(cuda)
        N.call("sph_grid_build_segments", N.ptr(pos), N.ptr(sup), N.ptr(seg), sets, None, None, 1 << 28, N.ptr(grids),
               N.ptr(status), N.stream_ptr())
        for k in {0, 1, 2, 3, 4, 5, 6, sets // 2, sets - 1} & set(range(sets)):
            a, b = int(off[k]), int(off[k + 1])
            scr = torch.empty(N.load().sph_grid_scratch_bytes(b - a) // 8 + 1, dtype=torch.int64, device=cuda)
            p, h = pos[a:b].clone(), sup[a:b].clone()
            N.call("sph_grid_build", N.ptr(p), N.ptr(h), b - a, None, None, 1 << 28, N.ptr(one), N.ptr(status),
                   N.ptr(scr), scr.numel() * 8, N.stream_ptr())
            assert torch.equal(one, grids[8 * k:8 * k + 8]), (sets, k)
        assert int(status.item()) == 0
    sets = 100000
    seg = torch.arange(0, 10 * sets + 1, 10, device=cuda)
    pos, sup, grids = torch.rand(10 * sets, 2, device=cuda), torch.full((10 * sets,), 0.1, device=cuda), i32(8 * sets)
    scr = torch.empty(N.load().sph_grid_scratch_bytes(10 * sets) // 8 + 1, dtype=torch.int64, device=cuda)
    taken = time_us(graph_of(lambda: N.call("sph_grid_build_segments", N.ptr(pos), N.ptr(sup), N.ptr(seg), sets, None,
                                            None, 1 << 28, N.ptr(grids), N.ptr(status), N.stream_ptr())))
    whole = time_us(graph_of(lambda: N.call("sph_grid_build", N.ptr(pos), N.ptr(sup), 10 * sets, None, None, 1 << 28,
                                            N.ptr(one), N.ptr(status), N.ptr(scr), scr.numel() * 8, N.stream_ptr())))
    assert taken < 35 * whole, (taken, whole)
