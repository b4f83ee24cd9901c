"""InterInsert in one launch (nodes in id order, waiting for their senders)
against the oracle: hubs with long insertion chains, tied distances, one slot
and the most slots per row, rows whose vectors do not fit shared memory, every
re-prune rule, and the dependency levels it reports."""
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
    rng = np.random.default_rng(31)
    if kind == "hub":  # every row near the first rows
        x = np.clip(np.rint(128 + 25 * rng.normal(size=(3000, 32))), 0, 255).astype(np.float32)
        x[:3] = 128.0 + np.arange(3)[:, None]
        return x
    if kind == "ties":
        return rng.integers(0, 3, (1200, 16)).astype(np.float32)
    if kind == "real":
        return ds.unit_mixture(2000, 44, 10, seed=6)[0]
    return ds.simplex_mixture(500, 960, 6, seed=6)[0]


@pytest.mark.parametrize("kind,R", [("hub", 32), ("hub", 63), ("hub", 4), ("ties", 20), ("ties", 1), ("real", 24),
                                    ("real", 40), ("long", 40)])
@pytest.mark.parametrize("link", ["nsg", "vamana", "clean", "ssg"])
def test_inter_insert_matches_oracle(ctx, link, kind, R):
    base = data(kind)
    ctx.upload_base(base)
    ctx.srand(1)
    ctx.init_random(10)
    ctx.nnd_refine(10, 24, 32, 4, 60)
    r = O.Rand(1)
    g = O.nndescent(base, O.init_random(base, 10, r), 10, 24, 32, 4, 60, r)
    if link == "nsg":
        st = ctx.nsg_refine(50, R, 400)
        want = O.nsg(base, g, 50, R, 400, r, out_w=R + 1500)
    elif link == "ssg":
        st = ctx.ssg_refine(80, R, 60.0, 2)
        want = O.ssg(base, g, 80, R, 60.0, 2, r, out_w=R + 1500)
    else:
        ctx.set_build_mode("clean" if link == "clean" else "compat")
        try:
            st = ctx.vamana_refine(50, R, 1.2)
        finally:
            ctx.set_build_mode("compat")
        want = O.vamana(base, g, 50, R, 1.2, r, clean=link == "clean")
    ids, dist, deg, _ = ctx.get_graph()
    assert st["levels"] >= 1
    assert np.array_equal(deg, want.deg)
    w = min(ids.shape[1], want.ids.shape[1])
    live = np.arange(w)[None, :] < deg[:, None]
    assert np.array_equal(ids[:, :w][live], want.ids[:, :w][live])
    assert np.array_equal(dist[:, :w][live].view(np.uint32), want.dist[:, :w][live].view(np.uint32))


@pytest.mark.parametrize("kind,R", [("hub", 60), ("hub", 61), ("real", 62)])
@pytest.mark.parametrize("link", ["nsg", "vamana", "clean", "ssg"])
def test_few_spare_slots_match_oracle(ctx, link, kind, R):
    """Rows with three, two and one spare slot: some of a batch's senders are
    copied ahead, the others where they are inserted."""
    test_inter_insert_matches_oracle(ctx, link, kind, R)


@pytest.mark.parametrize("link", ["nsg", "vamana"])
def test_repeated_builds_are_identical(ctx, link):
    """Rows beyond the L2 and many mutual edges (refused insertions): the rows
    must not depend on the order in which the vectors' copies land."""
    base = ds.unit_mixture(300000, 128, 300, seed=8)[0]
    ctx.upload_base(base)
    ctx.srand(1)
    ctx.init_random(10)
    ctx.nnd_refine(10, 32, 44, 4, 60)
    ids, dist, deg, _ = ctx.get_graph()
    first = None
    for _ in range(3):
        ctx.srand(2)
        ctx.set_graph(ids, deg, dist=dist)
        if link == "nsg":
            ctx.nsg_refine(50, 32, 300)
        else:
            ctx.vamana_refine(50, 32, 1.2)
        g = ctx.get_graph()
        rows = (g[0], g[1].view(np.uint32), g[2])
        if first is None:
            first = rows
        else:
            assert all(np.array_equal(x, y) for x, y in zip(first, rows))
