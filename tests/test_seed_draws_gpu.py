"""Centroid-entry seeds: one query and many, few ids and many per base row,
the entry row shorter and longer than L, and the rand() stream left where the
reference leaves it, across blocks of the generator."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from weavess_gb300 import Context
    return Context(0)


@pytest.mark.parametrize("n,deg", [(65, 7), (64, 63), (5000, 12), (70001, 40)])
@pytest.mark.parametrize("nq,L", [(1, 30), (2, 63), (400, 30), (37, 9)])
def test_centroid_seeds(ctx, n, deg, nq, L):
    rng = np.random.default_rng(n)
    ctx.upload_base(rng.normal(size=(n, 4)).astype(np.float32))
    ids = np.stack([rng.choice(n, deg, replace=False) for _ in range(8)])[np.arange(n) % 8].astype(np.uint32)
    g = O.Graph(ids, np.zeros(ids.shape, np.float32), np.full(n, deg, np.uint32), 5)
    ctx.upload_graph(ids, g.deg, 5)
    ctx.srand(9)
    r = O.Rand(9)
    for _ in range(2):
        assert np.array_equal(ctx.draw_seeds(nq, L, "centroid"), O.search_seeds(n, nq, g, L, r, "centroid"))
        assert ctx.rand() == r.next()
