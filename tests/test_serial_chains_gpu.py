"""Results that follow from one sequential chain: the centroid's FP32 column
sums (through the entry point and its search) at row counts around the tile,
and the mt19937 seeds of SEARCH_ENTRY_RAND at beams around the register sizes
and at batch sizes around the queries per block, against the host draw."""
import numpy as np
import pytest

import oracle as O
from weavess_gb300 import datasets as ds

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from weavess_gb300 import Context
    return Context(0)


@pytest.mark.parametrize("n,d", [(255, 16), (256, 20), (257, 36), (511, 96), (1500, 132)])
def test_centroid_entry_matches_oracle(ctx, n, d):
    base = (ds.unit_mixture(n, d, 5, seed=n)[0] * 1e3).astype(np.float32)
    ctx.upload_base(base)
    ctx.srand(1)
    ctx.init_random(8)
    ctx.nnd_refine(8, 12, 16, 4, 20)
    st = ctx.nsg_refine(20, 10, 60)
    r = O.Rand(1)
    g = O.nndescent(base, O.init_random(base, 8, r), 8, 12, 16, 4, 20, r)
    want = O.nsg(base, g, 20, 10, 60, r, out_w=200)
    assert st["ep"] == want.ep


@pytest.mark.parametrize("nq", [1, 31, 33, 304, 305, 700, 10000])
@pytest.mark.parametrize("L", [1, 31, 100, 128, 129, 226, 227, 256, 257, 454, 512, 513, 700])
def test_device_seeds_equal_host_seeds(ctx, nq, L):
    import torch
    n = 5000 if L % 2 else 701
    ctx.upload_base(np.zeros((n, 4), np.float32))
    d = torch.zeros((nq, L + 3), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ctx.srand(nq + L)
    ctx.draw_seeds_device(nq, L, d.data_ptr(), L + 3)
    nxt = ctx.rand()
    torch.cuda.synchronize()
    ctx.srand(nq + L)
    want = ctx.draw_seeds(nq, L, "rand")
    assert ctx.rand() == nxt
    got = d.cpu().numpy().astype(np.uint32)
    assert np.array_equal(got[:, :L], want)
    assert not got[:, L:].any()
