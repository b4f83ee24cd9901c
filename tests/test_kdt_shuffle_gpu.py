"""INIT_KDT's shuffled id lists and the splits of its active levels at sizes
about the 1024 steps and ids a block takes at once, against the oracle."""
import numpy as np
import pytest

import oracle as O
from golden_util import rows_equal
from weavess_gb300 import datasets as ds

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from weavess_gb300 import Context
    return Context(0)


@pytest.mark.parametrize("n,T,K", [(40, 1, 5), (1023, 2, 5), (1024, 3, 12), (1025, 2, 12), (2049, 3, 9), (5003, 9, 20),
                                   (700, 1100, 10)])
@pytest.mark.parametrize("ties", [False, True])
def test_forest_matches_oracle(ctx, n, T, K, ties):
    if ties:  # coordinates of four values: cuts fall between equal ids
        base = np.random.default_rng(n).integers(0, 4, (n, 16)).astype(np.float32)
        base += np.arange(n, dtype=np.float32)[:, None] / 64 * (np.arange(16) == 3)
    else:
        base, _ = ds.unit_mixture(n, 24, 6, seed=n, n_query=1)
    ctx.upload_base(base)
    ctx.srand(1)
    ctx.init_kdt(T, K, 3)
    g, _ = O.init_kdt(base, T, K, 3, O.Rand(1))
    ids, dist, deg, _ = ctx.get_graph()
    assert rows_equal(ids, dist, deg, g.ids, g.dist, g.deg) == 0
