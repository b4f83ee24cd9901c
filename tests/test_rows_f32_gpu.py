"""Real-valued rows in the reference's order, read by eight lanes at a time:
row lengths about the 32 and 64 dimensions of a step, few and many rows at
once, in the greedy route and its exact rerank.  Ids, counts and distance bits
against the oracle."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from weavess_gb300 import Context
    return Context(0)


def same_bits(dist, query, rows):
    want = np.stack([O.l2_rows(np.repeat(query[i:i + 1], rows.shape[1], 0), rows[i]) for i in range(len(query))])
    assert np.array_equal(dist.view(np.uint32), want.astype(np.float32).view(np.uint32))


@pytest.mark.parametrize("K", [8, 30])
@pytest.mark.parametrize("d", [4, 28, 32, 36, 60, 64, 68, 100, 132])
def test_route_matches_oracle(ctx, d, K):
    rng = np.random.default_rng(d)
    base = rng.normal(size=(900, d)).astype(np.float32)
    query = rng.normal(size=(33, d)).astype(np.float32)
    ctx.upload_base(base)
    ctx.srand(1)
    ctx.init_random(K)
    ctx.load_built_graph()
    ids, dist, deg, _ = ctx.get_graph()
    g = O.Graph(ids, dist, deg, 0)
    ctx.srand(3)
    res, dc, hc, dd = ctx.search(query, 45, 10, entry="rand", return_dist=True)
    want, wdc, whc = O.search(base, query, g, 45, O.Rand(3))
    assert np.array_equal(res, want) and (dc, hc) == (wdc, whc)
    same_bits(dd, query, base[res])
    ctx.set_precision("bf16")
    ctx.srand(3)
    res, dc, hc, dd = ctx.search(query, 45, 10, entry="rand", return_dist=True)
    same_bits(dd, query, base[res])
    ctx.set_precision("fp32")
