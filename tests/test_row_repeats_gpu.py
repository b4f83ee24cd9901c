"""Search graphs whose rows list an id twice, within 32 slots and further
apart, after and before a graph whose rows do not, on one context."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [9, 32, 50])
def test_rows_with_repeated_ids(w):
    from weavess_gb300 import Context
    ctx = Context(0)
    rng = np.random.default_rng(w)
    n = 1500
    base = rng.integers(0, 256, (n, 32)).astype(np.float32)
    query = rng.integers(0, 256, (60, 32)).astype(np.float32)
    ctx.upload_base(base)
    once = np.stack([rng.choice(n, w, replace=False) for _ in range(n)]).astype(np.uint32)
    near = once.copy()
    near[::3, w - 1] = near[::3, w - 3]  # repeats a few slots apart
    far = once.copy()
    far[:, -1] = far[:, 0]  # as far apart as the row allows
    for ids in (once, near, once, far):
        g = O.Graph(ids, np.zeros(ids.shape, np.float32), np.full(n, w, np.uint32), 0)
        ctx.upload_graph(ids, g.deg, 0)
        ctx.srand(4)
        res, dc, hc = ctx.search(query, 40, 10, entry="rand")
        want, wdc, whc = O.search(base, query, g, 40, O.Rand(4))
        assert np.array_equal(res, want) and (dc, hc) == (wdc, whc)
        ctx.set_expansion(2)  # the throughput form: no id twice among the results
        ctx.srand(4)
        res, _, _ = ctx.search(query, 40, 10, entry="rand")
        assert all(len(set(r)) == 10 for r in res.tolist())
        ctx.set_expansion(0)


@pytest.mark.parametrize("row,first,second", [(0, 0, 31), (777, 3, 4), (1499, 30, 31), (600, 33, 49), (5, 1, 40)])
def test_one_row_with_a_repeated_id(row, first, second):
    """A single row of 1,500 lists an id twice: its results must show that the
    second one was passed over."""
    from weavess_gb300 import Context
    ctx = Context(0)
    rng = np.random.default_rng(row)
    n, w = 1500, 50
    base = rng.integers(0, 256, (n, 32)).astype(np.float32)
    ids = np.stack([rng.choice(n, w, replace=False) for _ in range(n)]).astype(np.uint32)
    ids[row, second] = ids[row, first]
    query = base[np.r_[row, rng.integers(0, n, 60)]]  # the row itself is reached
    ctx.upload_base(base)
    g = O.Graph(ids, np.zeros(ids.shape, np.float32), np.full(n, w, np.uint32), 0)
    ctx.upload_graph(ids, g.deg, 0)
    ctx.srand(4)
    res, dc, hc = ctx.search(query, 40, 10, entry="rand")
    want, wdc, whc = O.search(base, query, g, 40, O.Rand(4))
    assert np.array_equal(res, want) and (dc, hc) == (wdc, whc)
