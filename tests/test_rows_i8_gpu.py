"""Searches over the byte copy of an integer base: every chunk count of a row
(d a multiple of 16 up to 256), the dimensions without one, integer and
real-valued queries on the same base, both traversals and both storages,
against the oracle's exact route and against the distances in FP64."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from weavess_gb300 import Context
    return Context(0)


@pytest.mark.parametrize("d", [16, 32, 48, 64, 80, 96, 128, 144, 240, 256, 100, 272])
def test_integer_rows_match_oracle(ctx, d):
    rng = np.random.default_rng(d)
    base = rng.integers(0, 256, (1500, d)).astype(np.float32)
    query = rng.integers(0, 256, (70, d)).astype(np.float32)
    query[::7] += 0.25  # real-valued queries take the ordered FP32 path
    ctx.upload_base(base)
    ctx.srand(1)
    ctx.init_random(12)
    ctx.nnd_refine(12, 24, 32, 4, 40)
    ctx.load_built_graph()
    ids, dist, deg, _ = ctx.get_graph()
    g = O.Graph(ids, dist, deg, 0)
    exact = lambda res: ((base[res].astype(np.float64) - query[:, None].astype(np.float64)) ** 2).sum(2)
    for storage in ("fp32", "bf16"):
        ctx.set_precision(storage)
        for E in (0, 2):
            ctx.set_expansion(E)
            ctx.srand(3)
            res, dc, hc, dd = ctx.search(query, 37, 10, entry="rand", return_dist=True)
            if storage == "fp32" and E == 0:
                want, wdc, whc = O.search(base, query, g, 37, O.Rand(3))
                assert np.array_equal(res, want) and (dc, hc) == (wdc, whc)
            e = exact(res)
            whole = np.arange(len(query)) % 7 != 0
            if d <= 256:  # integers below 2^24
                assert np.array_equal(dd[whole].astype(np.float64), e[whole])
            # d terms, each rounded, of a sum of e: d + 2 roundings of 2^-24
            assert np.all(np.abs(dd - e) <= (d + 2) * 2.0**-24 * (e + 2 * 255.0**2 * d))
        ctx.set_expansion(0)
    ctx.set_precision("fp32")


def test_upload_without_room_for_the_byte_copy():
    """A device whose memory holds the base but not its byte copy: the upload
    succeeds and the searches read the FP32 rows, with the same results."""
    torch = pytest.importorskip("torch")
    from weavess_gb300 import Context
    rng = np.random.default_rng(9)
    n, d = 2_000_000, 128
    base = rng.integers(0, 256, (n, d), dtype=np.uint8).astype(np.float32)
    query = rng.integers(0, 256, (40, d)).astype(np.float32)
    rows = rng.integers(0, n, (n, 6), dtype=np.uint32)
    out = []
    for tight in (True, False):
        ctx = Context(0)
        hold = None
        if tight:  # room for the rows, their norms and 96 MB; the byte copy takes 256
            free, _ = torch.cuda.mem_get_info()
            hold = torch.empty(free - (n * d * 4 + n * 4 + (96 << 20)), dtype=torch.uint8, device="cuda")
        ctx.upload_base(base)
        del hold
        torch.cuda.empty_cache()
        ctx.upload_graph(rows, np.full(n, 6, np.uint32))
        ctx.srand(1)
        out.append(ctx.search(query, 40, 10, entry="rand", return_dist=True))
        ctx.close()
    (i0, dc0, hc0, d0), (i1, dc1, hc1, d1) = out
    assert np.array_equal(i0, i1) and (dc0, hc0) == (dc1, hc1)
    assert np.array_equal(d0.view(np.uint32), d1.view(np.uint32))
