"""One-wait host reads (sph_read_i32) and what the searches read through them: word values,
their order, the limits, and the row offsets that a module search takes from its own scan."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("na,nb", [(1, 0), (9, 0), (1, 1), (15, 1), (16, 0)])
def test_words(cuda, na, nb):
    from pytorchsph_gb300 import _native as N
    a = torch.randint(-2**31, 2**31 - 1, (na,), dtype=torch.int32, device=cuda)
    b = torch.randint(-2**31, 2**31 - 1, (nb,), dtype=torch.int32, device=cuda)
    assert N.read_i32(a, b if nb else None) == a.tolist() + b.tolist()


def test_limits(cuda):
    from pytorchsph_gb300 import _native as N
    from pytorchsph_gb300.search import _total
    with pytest.raises(N.SPHError):
        N.read_i32(torch.zeros(16, dtype=torch.int32, device=cuda), torch.zeros(1, dtype=torch.int32, device=cuda))
    for v in (0, 5, 2**31, 2**33 + 7, 2**62):
        assert _total(torch.tensor([1, v], dtype=torch.int64, device=cuda)) == v


@pytest.mark.parametrize("n", [1, 33, 3000])
def test_module_search_offsets(cuda, n):
    from pytorchsph_gb300 import modules
    m = modules.neighborSearchModule()
    cfg = {"particle": {"support": 0.08}, "compute": {"maxNeighbors": 256, "precision": torch.float32, "device": "cuda"},
           "domain": {"virtualMin": [0.0, 0.0], "virtualMax": [1.0, 1.0]}}
    for p in m.getParameters():
        p.parseConfig(cfg)
    m.initialize(cfg, None)
    x = np.random.default_rng(n).uniform(0, 1, (n, 2)).astype(np.float32)
    st = {"fluidPosition": torch.from_numpy(x).cuda(), "fluidSupport": torch.full((n,), 0.08, device=cuda)}
    nb, _, _ = m.search(st, None)
    want = torch.searchsorted(nb[0].contiguous(), torch.arange(n + 1, device=cuda)).to(torch.int32)
    assert torch.equal(st["fluidNeighborOffsets"], want)
    st["fluidPosition"] = st["fluidPosition"] + float("nan")
    from pytorchsph_gb300 import _native as N
    with pytest.raises(N.SPHError):
        m.search(st, None)
