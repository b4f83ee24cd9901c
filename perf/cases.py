"""The work this framework is used for, as timed cases through its public API.

A case is a dict of plain values with a "kind" (what is called) and its sizes:

* ``search``   Context.search, host queries in, host ids and distances out;
* ``plan``     a captured plan on device buffers (``mode``: "rand" seeds, or
               "learned": the model's entry and beam per query), one replay;
* ``hnsw``     Context.search_hnsw over a layered graph;
* ``knn``      INIT_RANDOM and NN-Descent, from the vectors to the KNN graph;
* ``nsg``      the NSG link of a KNN graph (candidates, prune, InterInsert,
               connectivity);
* ``vamana``   INIT_RAND and two Vamana passes (alpha 1, then alpha);
* ``efanna``   INIT_KDT and the EFANNA refine;
* ``fit``      learn_fit: clusters, traces, training, calibration; then the
               trained model's predictions.

The data sets are the framework's own synthetic mixtures (datasets.py), drawn
on the GPU: ``int`` (integers in [0, 255]), ``unit`` (unit vectors),
``simplex`` (non-negative rows summing to 1).
"""
import numpy as np
import torch

from weavess_gb300 import Context


def listed():
    return [
        # one query of an interactive caller: latency, launches and copies
        {"name": "search_1_kgraph100k", "kind": "search", "data": "int", "n": 100_000, "d": 128, "graph": "knn",
         "nq": 1, "L": 100, "K": 10, "entry": "rand", "storage": "fp32", "E": 0},
        # a service's ordinary batch over a KGraph index (100k x 128, K = 20)
        {"name": "search_1000_kgraph100k", "kind": "search", "data": "int", "n": 100_000, "d": 128, "graph": "knn",
         "nq": 1000, "L": 100, "K": 10, "entry": "rand", "storage": "fp32", "E": 0},
        # unit vectors with fp8 candidates and the exact rerank, centroid
        # entry, a ragged batch and K
        {"name": "search_3001_unit96_fp8", "kind": "search", "data": "unit", "n": 120_001, "d": 96, "graph": "knn",
         "nq": 3001, "L": 250, "K": 17, "entry": "centroid", "storage": "fp8", "E": 0},
        # offline throughput: 10,000 queries of the exact FP32 traversal over an NSG index
        {"name": "plan_10000_nsg300k", "kind": "plan", "mode": "rand", "data": "int", "n": 300_000, "d": 128,
         "graph": "nsg", "nq": 10_000, "L": 200, "K": 10, "mixed": False, "storage": "fp32", "E": 0},
        # wide rows, every query its own k and beam, one launch
        {"name": "plan_20000_simplex960", "kind": "plan", "mode": "rand", "data": "simplex", "n": 30_000, "d": 960,
         "graph": "knn", "nq": 20_000, "L": 500, "K": 100, "mixed": True, "storage": "fp32", "E": 2},
        # the learned entry and beam with bf16 candidates
        {"name": "plan_10000_learned_bf16", "kind": "plan", "mode": "learned", "data": "int", "n": 200_000, "d": 128,
         "graph": "nsg", "nq": 10_000, "L": 256, "K": 10, "mixed": False, "storage": "bf16", "E": 3},
        # routing over a layered graph
        {"name": "hnsw_5000_100k", "kind": "hnsw", "data": "int", "n": 100_000, "d": 128, "nq": 5000, "L": 100,
         "K": 10},
        # the KGraph build (100k x 128: S 10, K 20, L 40, 8 rounds, R 100)
        {"name": "knn_int100k", "kind": "knn", "data": "int", "n": 100_000, "d": 128, "S": 10, "K": 20, "L": 40,
         "ITER": 8, "R": 100},
        # the NSG link of a K = 64 graph
        {"name": "nsg_int200k", "kind": "nsg", "data": "int", "n": 200_000, "d": 128, "K": 64, "L_refine": 64,
         "R_refine": 32, "C_refine": 500},
        # the Vamana pipeline on real-valued vectors
        {"name": "vamana_unit20k", "kind": "vamana", "data": "unit", "n": 20_011, "d": 96, "L_init": 64,
         "L_refine": 64, "R_refine": 32, "alpha": 1.2},
        # the EFANNA pipeline on real-valued vectors
        {"name": "efanna_unit60k", "kind": "efanna", "data": "unit", "n": 60_000, "d": 96, "trees": 8, "mlevel": 8,
         "S": 15, "K": 60, "L": 70, "ITER": 6, "R": 100},
        # training the entry and beam model on traces of its index
        {"name": "fit_20000_nsg100k", "kind": "fit", "data": "int", "n": 100_000, "d": 128, "nt": 20_000,
         "clusters": 64, "L_trace": 256, "epochs": 4, "batch": 1024},
    ]


def _log(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["search", "search", "plan", "plan", "hnsw", "knn", "nsg", "vamana", "efanna", "fit"])
    if kind == "search":
        data = rng.choice(["int", "unit"])
        L = _log(rng, 20, 300)
        return {"kind": kind, "data": data, "n": _log(rng, 5_000, 120_000), "d": 128 if data == "int" else 96,
                "graph": "knn", "nq": _log(rng, 1, 5000), "L": L, "K": min(L, rng.choice([1, 10, 17, 50])),
                "entry": rng.choice(["rand", "rand", "centroid"]), "storage": rng.choice(["fp32", "bf16", "fp8"]),
                "E": rng.choice([0, 0, 1, 2, 4])}
    if kind == "plan":
        mode = rng.choice(["rand", "rand", "learned"])
        if mode == "learned":
            return {"kind": kind, "mode": mode, "data": "int", "n": _log(rng, 30_000, 200_000), "d": 128,
                    "graph": "nsg", "nq": _log(rng, 100, 10_000), "L": 256, "K": 10, "mixed": False,
                    "storage": rng.choice(["fp32", "bf16"]), "E": rng.choice([0, 1, 2, 3])}
        data = rng.choice(["int", "unit", "simplex"])
        d = {"int": 128, "unit": 96, "simplex": 960}[data]
        L = _log(rng, 50, 500)
        return {"kind": kind, "mode": mode, "data": data,
                "n": _log(rng, 5_000, 30_000 if d == 960 else 200_000), "d": d, "graph": "knn",
                "nq": _log(rng, 10, 10_000), "L": L, "K": min(L, rng.choice([1, 10, 50, 100])),
                "mixed": rng.random() < 0.5, "storage": "fp32", "E": rng.choice([0, 0, 1, 2])}
    if kind == "hnsw":
        L = _log(rng, 20, 200)
        return {"kind": kind, "data": rng.choice(["int", "unit"]), "n": _log(rng, 5_000, 100_000), "d": 96, "L": L,
                "nq": _log(rng, 1, 5000), "K": min(L, 10)}
    if kind == "knn":
        K = rng.choice([20, 30, 64])
        return {"kind": kind, "data": rng.choice(["int", "unit"]), "n": _log(rng, 2_000, 100_000),
                "d": rng.choice([96, 128]), "S": rng.choice([10, 15, 20]), "K": K, "L": K + rng.randint(8, 24),
                "ITER": rng.randint(4, 8), "R": rng.choice([60, 100])}
    if kind == "nsg":
        return {"kind": kind, "data": rng.choice(["int", "int", "unit"]), "n": _log(rng, 5_000, 100_000), "d": 96,
                "K": rng.choice([32, 64]), "L_refine": rng.randint(40, 100), "R_refine": rng.choice([16, 32]),
                "C_refine": rng.choice([200, 500])}
    if kind == "vamana":
        return {"kind": kind, "data": rng.choice(["int", "unit"]), "n": _log(rng, 2_000, 20_000), "d": 96,
                "L_init": rng.randint(30, 64), "L_refine": rng.randint(40, 64), "R_refine": rng.choice([16, 32]),
                "alpha": rng.choice([1.2, 2.0])}
    if kind == "efanna":
        K = rng.randint(20, 60)
        return {"kind": kind, "data": rng.choice(["int", "unit"]), "n": _log(rng, 5_000, 60_000), "d": 96,
                "trees": rng.choice([4, 8]), "mlevel": rng.randint(4, 8), "S": rng.choice([10, 15]), "K": K,
                "L": K + rng.randint(5, 20), "ITER": rng.randint(4, 6), "R": rng.choice([60, 100])}
    return {"kind": "fit", "data": "int", "n": _log(rng, 20_000, 100_000), "d": 128, "nt": _log(rng, 3_000, 20_000),
            "clusters": rng.choice([16, 64]), "L_trace": rng.choice([128, 256]), "epochs": rng.randint(2, 4),
            "batch": rng.choice([256, 1024])}


# ---------------------------------------------------------------- inputs
def _mixture(data, d, sizes, seed):
    """Samples of one mixture, drawn on the GPU: a host float32 array per size."""
    g = torch.Generator(device="cuda").manual_seed(seed * 1000 + 7)
    kw = dict(generator=g, device="cuda")
    parts = {"int": 64, "unit": 1000, "simplex": 512}[data]
    cent = torch.rand(parts, d, **kw) * 255.0 if data == "int" else torch.randn(parts, d, **kw)
    if data == "unit":
        cent = torch.nn.functional.normalize(cent)
    out = []
    for n in sizes:
        u = cent[torch.randint(parts, (n,), **kw)]
        z = torch.randn(n, d, **kw)
        if data == "int":
            x = (u + 20.0 * z).round().clamp(0.0, 255.0)
        elif data == "simplex":
            x = (u + 0.5 * z).clamp(min=0.0)
            x = x / x.sum(1, keepdim=True).clamp(min=1e-12)
        else:  # cosine 0.7 to the direction, one tenth isotropic
            v = torch.nn.functional.normalize(z - (z * u).sum(1, keepdim=True) * u)
            x = 0.7 * u + (1.0 - 0.7 * 0.7) ** 0.5 * v
            x = torch.where(torch.rand(n, 1, **kw) < 0.1, z, x)
            x = torch.nn.functional.normalize(x)
        out.append(x.cpu().numpy())
    return out


def _knn(ctx, K=20, S=10, L=40, ITER=8, R=100):
    ctx.init_random(S)
    ctx.nnd_refine(S, K, L, ITER, R)


def _index(case, base):
    """A context with the case's vectors and search graph."""
    ctx = Context(0)
    ctx.upload_base(base)
    ctx.srand(1)
    if case["graph"] == "knn":
        _knn(ctx)
    else:
        _knn(ctx, K=40, S=15, L=56, ITER=6)
        ctx.nsg_refine(56, 32, 300)
    ctx.load_built_graph()
    return ctx


def _layered(ctx, base, seed):
    """INDEX_HNSW words: layer 0 the built graph's rows, levels by HNSW's rule
    (m = 16), each upper layer the exact 16-NN graph of its nodes."""
    ids, _, deg, _ = ctx.get_graph()
    n, m = base.shape[0], 16
    rng = np.random.default_rng(seed)
    level = np.minimum(rng.geometric(1 - 1 / m, size=n) - 1, 6)
    top = int(level.max())
    start = np.zeros(n + 1, np.int64)  # of each node's record, after the two header words
    cols = np.arange(ids.shape[1])[None, :]
    rec = [deg.astype(np.int64) + 3]
    upper = []
    for lv in range(1, top + 1):
        at = np.flatnonzero(level >= lv)
        k = min(m, len(at) - 1)
        size = np.zeros(n, np.int64)
        if k > 0:
            x = torch.from_numpy(base[at]).cuda()
            near = torch.cdist(x, x).topk(k + 1, largest=False).indices.cpu().numpy()
            keep = np.argsort(near == np.arange(len(at))[:, None], axis=1, kind="stable")[:, :k]
            near = at[np.take_along_axis(near, keep, 1)]
        else:
            near = np.zeros((len(at), 0), np.int64)
        size[at] = k + 1
        upper.append((at, near))
        rec.append(size)
    start[1:] = np.cumsum(sum(rec))
    w = np.zeros(2 + start[-1], np.uint32)
    w[0], w[1] = np.flatnonzero(level == top)[0], top
    s = start[:-1] + 2
    w[s], w[s + 1], w[s + 2] = np.arange(n), level + 1, deg
    live = cols < deg[:, None]
    w[(s[:, None] + 3 + cols)[live]] = ids[live]
    off = s + rec[0]
    for (at, near), size in zip(upper, rec[1:]):
        w[off[at]] = near.shape[1]
        w[off[at][:, None] + 1 + np.arange(near.shape[1])[None, :]] = near
        off = off + size
    return w


def prepare(case, seed):
    kind, n, d = case["kind"], case["n"], case["d"]
    if kind in ("search", "plan", "hnsw"):
        learned = case.get("mode") == "learned"
        base, query, train = _mixture(case["data"], d, (n, case["nq"], 4000 if learned else 1), seed)
        st = {"case": case, "query": query}
        if kind == "hnsw":
            ctx = Context(0)
            ctx.upload_base(base)
            ctx.srand(1)
            _knn(ctx, K=32, L=44)
            ctx.load_hnsw(_layered(ctx, base, seed))
            return dict(st, ctx=ctx)
        ctx = _index(case, base)
        if learned:
            ctx.learn_fit(train, clusters=64, L_trace=256, L_max=case["L"], list_len=case["L"], epochs=3, batch=256,
                          seed=seed & 0xffff)
        ctx.set_precision(case["storage"])
        ctx.set_expansion(case["E"])
        if kind == "search":
            return dict(st, ctx=ctx)
        nq, K, L = case["nq"], case["K"], case["L"]
        dq = torch.from_numpy(query).cuda()
        out = torch.full((nq, K), -1, dtype=torch.int32, device="cuda")
        dist = torch.zeros((nq, K), dtype=torch.float32, device="cuda")
        dL = dK = None
        if case["mixed"]:
            r = np.random.default_rng(seed)
            hK = np.minimum(K, r.choice([1, 10, 50, 100], size=nq))
            hL = np.maximum(hK, r.integers(min(10, L), L + 1, size=nq))
            dK, dL = (torch.from_numpy(v.astype(np.int32)).cuda() for v in (hK, hL))
        torch.cuda.synchronize()
        plan = ctx.plan(nq, K, dq.data_ptr(), out.data_ptr(), L_max=0 if learned else L, mode=case["mode"],
                        d_L=dL.data_ptr() if dL is not None else 0, d_K=dK.data_ptr() if dK is not None else 0,
                        d_out_dist=dist.data_ptr())
        return dict(st, ctx=ctx, plan=plan, dq=dq, out=out, dist=dist, dL=dL, dK=dK)
    if kind == "fit":
        base, train, held = _mixture(case["data"], d, (n, case["nt"], 1000), seed)
        ctx = _index({"graph": "nsg"}, base)
        return {"case": case, "ctx": ctx, "train": train, "held": held}
    (base,) = _mixture(case["data"], d, (n,), seed)
    ctx = Context(0)
    st = {"case": case, "ctx": ctx}
    if kind == "nsg":
        ctx.upload_base(base)
        ctx.srand(1)
        _knn(ctx, K=case["K"], S=20, L=case["K"] + 16, ITER=6)
        ids, dist, deg, _ = ctx.get_graph()
        return dict(st, ids=ids, dist=dist, deg=deg)
    return dict(st, base=base)


# ---------------------------------------------------------------- the calls
def _graph(ctx, width):
    """The built graph.  The connectivity pass may lengthen some rows beyond
    `width`: those rows' further entries come apart, at a size that does not
    depend on the data."""
    ids, dist, deg, ep = ctx.get_graph()
    out = {"ids": ids.view(np.int32)[:, :width], "dist": dist[:, :width], "deg": deg.view(np.int32), "ep": ep}
    more = np.zeros((ids.shape[0] // 16 + 64, 64), np.int32)
    long = np.flatnonzero(deg > width)[:more.shape[0]]
    more[:len(long), :ids.shape[1] - width] = ids.view(np.int32)[long, width:width + 64]
    return dict(out, more=more)


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    ctx.srand(1)
    if kind == "search":
        ids, dc, hc, dist = ctx.search(state["query"], case["L"], case["K"], entry=case["entry"], return_dist=True)
        return {"ids": ids.view(np.int32), "dist": dist, "dist_count": dc, "hop_count": hc}
    if kind == "plan":
        state["plan"].run(case["nq"])
        dc, hc = state["plan"].wait()
        return {"ids": state["out"], "dist": state["dist"], "dist_count": dc, "hop_count": hc}
    if kind == "hnsw":
        ids, dist, dc, hc = ctx.search_hnsw(state["query"], case["L"], case["K"], return_dist=True)
        return {"ids": ids.view(np.int32), "dist": dist, "dist_count": dc, "hop_count": hc}
    if kind == "fit":
        rep = ctx.learn_fit(state["train"], clusters=case["clusters"], L_trace=case["L_trace"], L_max=256,
                            list_len=256, epochs=case["epochs"], batch=case["batch"])
        cluster, prob, log2L = ctx.learn_predict(state["held"])
        return {"loss": [rep["loss_ce"], rep["loss_mse"]], "margin": rep["margin"], "labelled": rep["labelled"],
                "agreement": rep["val_agreement"], "cluster": cluster.view(np.int32), "prob": prob, "log2L": log2L}
    if kind == "nsg":
        ctx.set_graph(state["ids"], state["deg"], dist=state["dist"])
        ctx.nsg_refine(case["L_refine"], case["R_refine"], case["C_refine"])
        return _graph(ctx, case["R_refine"])
    ctx.upload_base(state["base"])
    if kind == "knn":
        ctx.init_random(case["S"])
        ctx.nnd_refine(case["S"], case["K"], case["L"], case["ITER"], case["R"])
    elif kind == "vamana":
        ctx.init_rand(case["L_init"])
        ctx.vamana_refine(case["L_refine"], case["R_refine"], 1.0)
        ctx.vamana_refine(case["L_refine"], case["R_refine"], case["alpha"])
    else:
        ctx.init_kdt(case["trees"], case["K"], case["mlevel"])
        ctx.efanna_refine(case["S"], case["K"], case["L"], case["ITER"], case["R"])
    return _graph(ctx, case["R_refine"] if kind == "vamana" else case["K"])


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Bytes: the inputs read once (of a search, the rows it looks at, each at
    most once), the outputs written once.  Operations: two per dimension of
    every distance; a search looks at about half a row's neighbours anew per
    expansion and expands about its beam, a link's candidate search the same,
    NN-Descent joins about S new with 3 S other ids per node and round."""
    kind, n, d = case["kind"], case["n"], case["d"]
    if kind in ("search", "plan", "hnsw"):
        nq, K = case["nq"], case["K"]
        L = case["L"] * (0.4 if case.get("mode") == "learned" else 0.55 if case.get("mixed") else 1.0)
        width = 32 if kind == "hnsw" or case.get("graph") == "nsg" else 20
        size = {"fp32": 4, "bf16": 2, "fp8": 1}[case.get("storage", "fp32")]
        dists = nq * min(n, L + L * width / 2)
        rows, hops = min(n, dists), min(n, nq * L)
        return {"bytes": rows * d * size + hops * width * 4 + nq * d * 4 + nq * K * 8, "flops": dists * 2 * d}
    if kind == "fit":
        steps = case["epochs"] * (case["nt"] * 9 // 10 // case["batch"])
        weights = d * 256 + 256 * 256 + 256 * (case["clusters"] + 1)
        search = case["nt"] * case["L_trace"] * 16 * 2 * d
        return {"bytes": n * d * 4 + n * 32 * 4 + case["nt"] * d * 4,
                "flops": search + 9 * n * case["clusters"] * 2 * d + steps * case["batch"] * weights * 6}
    if kind == "nsg":
        dists = n * (case["L_refine"] * case["K"] / 2 + case["R_refine"] * 100)
        return {"bytes": n * d * 4 + n * case["K"] * 8 + n * case["R_refine"] * 8, "flops": dists * 2 * d}
    if kind == "vamana":
        dists = 2 * n * (case["L_refine"] * 16 + case["R_refine"] * 100)
        return {"bytes": n * d * 4 + n * case["R_refine"] * 8, "flops": dists * 2 * d}
    dists = n * case["ITER"] * 3 * case["S"] * case["S"]
    if kind == "efanna":
        dists += n * case["trees"] * 100
    return {"bytes": n * d * 4 + n * case["K"] * 8, "flops": dists * 2 * d}


def exact(case, seed):
    """None: the outputs are ids, counts and the distances of the ids found,
    which follow from the algorithm's own order and not from a formula."""
    return None
