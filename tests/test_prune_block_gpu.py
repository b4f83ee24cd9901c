"""The prune with a block per node against the oracle where it can go wrong:
few distinct distances (every tie goes to the std::sort replica), pools just
below and above the sort's sizes and beyond the largest, one slot and the most
slots per row, a small examination bound, rows too long for shared memory, a
base whose rows repeat, short pools."""
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
    rng = np.random.default_rng(23)
    if kind == "ties":
        return rng.integers(0, 3, (1500, 16)).astype(np.float32)
    if kind == "repeats":
        x = ds.int_mixture(700, 32, 4, seed=9)[0]
        return np.concatenate([x, x[:500]])
    if kind == "real":
        return ds.unit_mixture(1500, 36, 20, seed=4)[0]
    if kind == "long":
        return ds.simplex_mixture(600, 960, 8, seed=4)[0]
    return ds.int_mixture(6000, 48, 4, seed=9)[0]


def same(ctx, g):
    ids, dist, deg, ep = ctx.get_graph()
    assert np.array_equal(deg, g.deg)
    w = min(ids.shape[1], g.ids.shape[1])
    live = np.arange(w)[None, :] < deg[:, None]
    assert np.array_equal(ids[:, :w][live], g.ids[:, :w][live])
    assert np.array_equal(dist[:, :w][live].view(np.uint32), g.dist[:, :w][live].view(np.uint32))


@pytest.mark.parametrize("link,kind,L,R,C", [
    ("nsg", "ties", 40, 32, 200), ("nsg", "repeats", 30, 16, 100), ("nsg", "real", 50, 32, 500),
    ("nsg", "int", 60, 32, 500), ("nsg", "int", 400, 24, 3000), ("nsg", "int", 40, 1, 30), ("nsg", "real", 40, 63, 5000),
    ("nsg", "long", 40, 20, 300), ("vamana", "ties", 40, 32, 0), ("vamana", "repeats", 30, 16, 0),
    ("vamana", "real", 60, 40, 0), ("vamana", "int", 300, 63, 0), ("vamana", "long", 30, 12, 0),
    ("vamana", "int", 8, 60, 0), ("clean", "ties", 40, 32, 0), ("clean", "repeats", 30, 16, 0),
    ("clean", "real", 60, 24, 0), ("clean", "int", 100, 32, 0), ("ssg", "ties", 60, 32, 0), ("ssg", "real", 100, 40, 0),
    ("ssg", "int", 300, 63, 0), ("ssg", "repeats", 50, 1, 0)])
def test_prune_matches_oracle(ctx, link, kind, L, R, C):
    base = data(kind)
    ctx.upload_base(base)
    ctx.srand(1)
    ctx.init_random(10)
    ctx.nnd_refine(10, 20, 32, 4, 40)
    r = O.Rand(1)
    g = O.nndescent(base, O.init_random(base, 10, r), 10, 20, 32, 4, 40, r)
    if link == "nsg":
        ctx.nsg_refine(L, R, C)
        same(ctx, O.nsg(base, g, L, R, C, r, out_w=R + 1500))
    elif link == "ssg":
        ctx.ssg_refine(L, R, 60.0, 3)
        same(ctx, O.ssg(base, g, L, R, 60.0, 3, r, out_w=R + 1500))
    else:
        ctx.set_build_mode("clean" if link == "clean" else "compat")
        try:
            ctx.vamana_refine(L, R, 1.2)
        finally:
            ctx.set_build_mode("compat")
        same(ctx, O.vamana(base, g, L, R, 1.2, r, clean=link == "clean"))
