"""Real-valued rows in the reference's order, read by eight lanes at a time:
row lengths about the 32 and 64 dimensions of a step, few and many rows at
once, in the greedy route, its exact rerank and the layered route, whose lists
here also hold an id twice.  Ids, counts and distance bits against the
oracle."""
import numpy as np
import pytest

import oracle as O
from weavess_gb300 import datasets as ds

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


@pytest.mark.parametrize("router", ["hnsw", "nsw"])
@pytest.mark.parametrize("kind,d", [("int", 128), ("int", 48), ("int", 20), ("real", 36), ("real", 128)])
def test_layered_route_with_repeated_ids(ctx, kind, d, router):
    rng = np.random.default_rng(d)
    n = 1200
    if kind == "int":
        base, query = ds.int_mixture(n, d, 8, seed=5, n_query=40)
        query[::5] += 0.25  # a real-valued query on integer rows
    else:
        base, query = rng.normal(size=(n, d)).astype(np.float32), rng.normal(size=(40, d)).astype(np.float32)
    for repeats in (False, True):
        words = [3, 1]
        for v in range(n):
            layers = 2 if v % 16 == 3 else 1
            words += [v, layers]
            for lv in range(layers):
                pool = np.arange(n) if lv == 0 else np.arange(3, n, 16)
                row = rng.choice(pool, 36 if lv == 0 else 8, replace=False).tolist()
                if repeats:
                    row = row[:20] + row[5:9] + row[20:] + row[:3]
                words += [len(row)] + row
        words = np.array(words, np.uint32)
        ctx.upload_base(base)
        ctx.load_hnsw(words)
        for L in (10, 70):
            res, dist, dc, hc = ctx.search_hnsw(query, L, 10, router=router, return_dist=True)
            want, wdc, whc = O.search_hnsw(base, query, words, L, router=router)
            assert np.array_equal(res, want) and (dc, hc) == (wdc, whc)
            same_bits(dist, query, base[res])


@pytest.mark.parametrize("d", [8, 12, 16, 20])
def test_short_rows_match_oracle(ctx, d):
    """Rows about the length up to which a lane reads a whole row."""
    test_route_matches_oracle(ctx, d, 24)


@pytest.mark.parametrize("kind,d", [("int", 64), ("int", 80), ("int", 128), ("int", 144), ("int", 256),
                                    ("real", 188), ("real", 192)])
def test_layered_route_every_way_of_reading_rows(ctx, kind, d):
    """Byte rows (integer rows of 65 to 128 dimensions, integer and real-valued
    queries in one batch), a lane per row, eight lanes per row."""
    rng = np.random.default_rng(d)
    n = 1200
    if kind == "int":
        base, query = ds.int_mixture(n, d, 8, seed=5, n_query=40)
    else:
        base, query = rng.normal(size=(n, d)).astype(np.float32), rng.normal(size=(40, d)).astype(np.float32)
    words = [3, 1]
    for v in range(n):
        upper = v % 16 == 3
        words += [v, 1 + upper, 36] + rng.choice(n, 36, replace=False).tolist()
        if upper:
            words += [8] + rng.choice(np.arange(3, n, 16), 8, replace=False).tolist()
    words = np.array(words, np.uint32)
    ctx.upload_base(base)
    ctx.load_hnsw(words)
    for real_at in (None, 1, 0):
        q = query.copy()
        if real_at is not None:
            q[real_at::5] += 0.25
        res, dist, dc, hc = ctx.search_hnsw(q, 40, 10, return_dist=True)
        want, wdc, whc = O.search_hnsw(base, q, words, 40, router="hnsw")
        assert np.array_equal(res, want) and (dc, hc) == (wdc, whc)
        same_bits(dist, q, base[res])
