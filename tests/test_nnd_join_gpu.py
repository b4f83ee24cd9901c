"""The local join's offers and their order-free application, against the
single-threaded oracle: distances that tie (those targets are replayed in the
reference's order), a hub that takes more offers than a warp's or a block's
shared memory holds, lists beyond one tile, the widest and narrowest integer
rows, init rows whose distances are not those of their ids, and joins in
chunks.  Rows must be identical: ids in order and distance bits."""
import numpy as np
import pytest

import oracle as O
from weavess_gb300 import datasets as ds

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from weavess_gb300 import Context
    return Context(0)


def data(kind):
    rng = np.random.default_rng(17)
    if kind == "ties":  # few distinct distances
        return rng.integers(0, 4, (2500, 16)).astype(np.float32)
    if kind == "hub":  # row 0 is the centre: in every list, offered to by every node
        x = np.clip(np.rint(128 + 30 * rng.normal(size=(4000, 32))), 0, 255).astype(np.float32)
        x[0] = 128.0
        return x
    if kind == "hub_real":
        x = rng.normal(size=(4000, 24)).astype(np.float32)
        x[0] = 0.0
        return x
    if kind in ("long", "longest"):  # real-valued rows whose tiles are smaller
        return rng.normal(size=(700, 200 if kind == "long" else 1000)).astype(np.float32)
    if kind == "wide":  # integer rows of 256 dimensions
        return ds.int_mixture(1500, 256, 6, seed=3)[0]
    if kind == "odd":  # integer data without byte rows (d not a multiple of 16)
        return ds.int_mixture(1500, 20, 6, seed=3)[0]
    return ds.int_mixture(1500, 16, 6, seed=3)[0]


def same(ctx, g):
    ids, dist, deg, _ = ctx.get_graph()
    assert np.array_equal(deg, g.deg)
    live = np.arange(ids.shape[1])[None, :] < deg[:, None]
    assert np.array_equal(ids[live], g.ids[:, :ids.shape[1]][live])
    assert np.array_equal(dist[live].view(np.uint32), g.dist[:, :ids.shape[1]][live].view(np.uint32))


@pytest.mark.parametrize("kind,S,K,L,R,cap", [
    ("ties", 10, 20, 40, 60, None), ("ties", 10, 20, 40, 60, "20000"), ("hub", 12, 20, 40, 100, None),
    ("hub_real", 12, 20, 40, 100, None), ("wide", 10, 20, 33, 40, None), ("odd", 10, 20, 40, 60, None),
    ("narrow", 30, 60, 256, 150, None), ("narrow", 1, 1, 1, 1, None), ("long", 20, 20, 40, 60, None),
    ("longest", 20, 20, 40, 60, None)])
def test_join_matches_oracle(ctx, kind, S, K, L, R, cap, monkeypatch):
    if cap:
        monkeypatch.setenv("WV_NND_OFFER_CAP", cap)
    base = data(kind)
    ctx.upload_base(base)
    ctx.srand(1)
    ctx.init_random(S)
    st = ctx.nnd_refine(S, K, L, 5, R)
    assert cap is None or st["chunks"] > 5
    r = O.Rand(1)
    same(ctx, O.nndescent(base, O.init_random(base, S, r), S, K, L, 5, R, r))
    assert ctx.rand() == r.next()


def test_stale_init_distances(ctx):
    """Init rows may carry other distances than those of their ids."""
    base = data("narrow")
    r = O.Rand(1)
    g0 = O.init_random(base, 10, r)
    g0.dist[::3] += 7.5
    ctx.upload_base(base)
    ctx.srand(1)
    ctx.rand()  # the init's draw
    ctx.set_graph(g0.ids, g0.deg, dist=g0.dist)
    ctx.nnd_refine(10, 20, 30, 4, 40)
    same(ctx, O.nndescent(base, g0, 10, 20, 30, 4, 40, r))


@pytest.mark.parametrize("kind", ["narrow", "hub", "long"])
def test_join_in_chunks_of_list_entries(ctx, kind, monkeypatch):
    """A join whose lists exceed a launch's limit runs in chunks of nodes."""
    monkeypatch.setenv("WV_NND_LIST_CAP", "8000")
    base = data(kind)
    ctx.upload_base(base)
    ctx.srand(1)
    ctx.init_random(10)
    st = ctx.nnd_refine(10, 20, 40, 5, 60)
    assert st["chunks"] > 4  # joins
    r = O.Rand(1)
    same(ctx, O.nndescent(base, O.init_random(base, 10, r), 10, 20, 40, 5, 60, r))
    assert ctx.rand() == r.next()
