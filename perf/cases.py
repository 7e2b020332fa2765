"""The calls that a user of this library makes, at the sizes they make them.

A service keeps an index on the GPU (rows, attribute columns, and for graph
search the HNSW lists) and answers batches of filtered nearest-neighbour
queries against it. A case names the index, the call and the batch; the seed
draws what changes from call to call, the queries and the filters' constants.
Rows come from the library's own stand-in for SIFT (a Gaussian mixture,
centres U[0, 128], sigma 20: rounded to 0..255, or left as real numbers like
an embedding), columns are a category 0..9 and a price U[0, 1000).
"""
import functools
import math
import random

import numpy as np
import torch

from paves_b200 import _lib, datagen
from paves_b200.hnsw import Hnsw
from paves_b200.index import GpuIndex
from paves_b200.pred import And, Cmp, In, Not, Or, concat, eval_numpy
from paves_b200.router import Router, routed_batch
from paves_b200.stream import Stream

PRICE, CATEGORY = datagen.COL_PRICE, datagen.COL_CATEGORY
PRECISION = {"fp32": _lib.FV_GPU_PREC_FP32, "sq8": _lib.FV_GPU_PREC_SQ8,
             "bf16": _lib.FV_GPU_PREC_BF16, "fp8": _lib.FV_GPU_PREC_FP8}
ELEMENT = {"fp32": 4, "sq8": 2, "bf16": 2, "fp8": 1}
STREAM_BATCH, STREAM_K = 512, 100
ROUTER_FILE = "paves_b200/router_1m128.npz"


def listed():
    fp32 = {"call": "brute", "precision": "fp32"}
    small = {"rows": 100_000, "dim": 128, "values": "int"}
    million = {"rows": 1_000_000, "dim": 128, "values": "int"}
    return [
        # one user, one query, a small table: nothing but latency
        {"name": "one_query_100k", **fp32, **small, "batch": 1, "k": 10, "filter": "both", "sel": 0.02},
        # the exact search of a small table for a whole evaluation set
        {"name": "exact_256_100k", **fp32, **small, "batch": 256, "k": 10, "filter": "both", "sel": 0.02},
        # one interactive query over a million rows: the rows stream once
        {"name": "exact_1_1m", **fp32, **million, "batch": 1, "k": 10, "filter": "range", "sel": 0.7},
        # real-valued rows, exact answers, several filters in one batch
        {"name": "exact_64_1m_real", **fp32, "rows": 1_000_000, "dim": 128, "values": "real",
         "batch": 64, "k": 10, "filter": "mixed", "sel": 0.3},
        # wide embeddings, an odd batch, a longer result list
        {"name": "exact_33_200k_d384", **fp32, "rows": 200_003, "dim": 384, "values": "real",
         "batch": 33, "k": 50, "filter": "or", "sel": 0.3},
        # the headline batch: routed, one filter of 10 % for 64 queries
        {"name": "routed_64_1m", "call": "routed", "precision": "bf16", **million, "batch": 64,
         "k": 10, "filter": "in", "sel": 0.1},
        # a selective filter: 1 % of the rows pass
        {"name": "selective_64_1m", "call": "brute", "precision": "bf16", **million, "batch": 64,
         "k": 10, "filter": "range", "sel": 0.01},
        # a large batch with several filters
        {"name": "bf16_512_1m", "call": "brute", "precision": "bf16", **million, "batch": 512,
         "k": 10, "filter": "mixed", "sel": 0.3},
        # filtered graph search of concurrent queries
        {"name": "graph_64_1m", "call": "graph", "precision": "bf16", **million, "batch": 64,
         "k": 64, "filter": "in", "sel": 0.1},
        # a micro-batch of the arrival stream, a filter and a k per query
        {"name": "stream_29_2m", "call": "stream", "precision": "fp8", "rows": 2_000_000, "dim": 96,
         "values": "int", "batch": 29, "k": 100, "filter": "each", "sel": 0.0},
        # the stream's largest micro-batch
        {"name": "stream_512_2m", "call": "stream", "precision": "fp8", "rows": 2_000_000, "dim": 96,
         "values": "int", "batch": 512, "k": 100, "filter": "each", "sel": 0.0},
        # building a table's graph
        {"name": "build_60k", "call": "build", "precision": "bf16", "rows": 60_000, "dim": 128,
         "values": "int", "batch": 0, "k": 16, "filter": "none", "sel": 1.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["brute"] * 5 + ["graph", "graph", "stream", "routed", "build"])
    values = rng.choice(["int", "real"])
    if call == "build":
        return {"call": call, "precision": "bf16" if values == "int" else "fp32",
                "rows": _log(rng, 2000, 60_000 if values == "int" else 20_000),
                "dim": rng.choice([96, 100, 128]), "values": values, "batch": 0,
                "k": rng.choice([8, 16]), "filter": "none", "sel": 1.0}
    flt = rng.choice(["none", "range", "range", "in", "both", "or", "mixed"])
    sel = round(math.exp(rng.uniform(math.log(0.001), math.log(0.95))), 4)
    batch = _log(rng, 1, 512)
    if call == "stream":
        precision = rng.choice(["fp8", "bf16"])
        return {"call": call, "precision": precision, "rows": _log(rng, 50_000, 2_000_000),
                "dim": rng.choice([96, 128] if precision == "bf16" else [96, 100]),
                "values": "int", "batch": batch, "k": STREAM_K, "filter": "each", "sel": 0.0}
    if call == "routed":
        return {"call": call, "precision": rng.choice(["bf16", "fp32"]),
                "rows": _log(rng, 50_000, 1_000_000), "dim": 128, "values": "int",
                "batch": batch, "k": 10, "filter": flt, "sel": sel}
    if call == "graph":
        return {"call": call, "precision": "bf16", "rows": _log(rng, 20_000, 1_000_000),
                "dim": rng.choice([96, 128]), "values": "int", "batch": max(1, batch // 2),
                "k": rng.choice([16, 32, 64, 100, 128, 256]), "filter": flt,
                "sel": max(sel, 0.01)}
    dim = rng.choice([64, 96, 100, 128, 128, 200, 384])
    return {"call": call, "precision": rng.choice(["fp32", "fp32", "bf16", "bf16", "fp8", "sq8"]),
            "rows": _log(rng, 20_000, min(1_000_000, 100_000_000 // dim)), "dim": dim,
            "values": values, "batch": batch, "k": _log(rng, 1, 200), "filter": flt, "sel": sel}


# ------------------------------------------------------------- the service
def _centers(dim, n):
    return np.random.default_rng(datagen.SEED).uniform(0.0, 128.0, (n, dim)).astype(np.float32)


def _mixture(gen, centers, n, values):
    """n draws of the mixture on the GPU, in blocks -> host array."""
    c = torch.from_numpy(centers).cuda()
    out = np.empty((n, c.shape[1]), np.float32)
    for s in range(0, n, 1 << 20):
        m = min(1 << 20, n - s)
        comp = torch.randint(0, c.shape[0], (m,), generator=gen, device="cuda")
        x = torch.randn((m, c.shape[1]), generator=gen, device="cuda") * 20.0 + c[comp]
        if values == "int":
            x = x.clamp(0.0, 255.0).round()
        out[s:s + m] = x.cpu().numpy()
    return out


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


_kept = {}  # what the service has loaded: the last few indexes


def _service(case):
    """The loaded index (and its graph, stream, router) that a program keeps
    for as long as it answers queries."""
    graph = case["call"] in ("graph", "routed")
    key = (case["rows"], case["dim"], case["values"], case["precision"], graph)
    s = _kept.pop(key, None)
    if s is None:
        while len(_kept) >= 6:
            old = _kept.pop(next(iter(_kept)))
            if "stream" in old:
                old["stream"].close()
            old["index"].close()
        n = case["rows"]
        # (tables searched through a graph: clusters of about 2000 rows, so that
        # no row is a hub whose surplus links the builder keeps in any order)
        centers = _centers(case["dim"], max(64, n // 2000) if graph else 256 if n > 1_000_000 else 64)
        rows = _mixture(_gen(datagen.SEED + 1), centers, n, case["values"])
        rng = np.random.default_rng(datagen.SEED + 3)
        cols = np.stack([rng.integers(0, 10, n).astype(np.float64),
                         rng.uniform(0.0, 1000.0, n).astype(np.float32).astype(np.float64)])
        s = {"centers": centers, "rows": rows, "cols": cols}
        l0 = None
        if graph:
            s["hnsw"] = Hnsw(rows, 16, builder="gpu")
            l0 = s["hnsw"].l0
        s["index"] = GpuIndex(rows, cols, l0=l0, precision=PRECISION[case["precision"]], device=0)
    if case["call"] == "stream" and "stream" not in s:
        tune = _mixture(_gen(datagen.SEED + 2), s["centers"], STREAM_BATCH, case["values"])
        s["stream"] = Stream(s["index"], STREAM_BATCH, STREAM_K, tune)
    if case["call"] == "routed" and "router" not in s:
        z = np.load(ROUTER_FILE)
        s["router"] = Router(z["centroids"].astype(np.float32), device=0)
        s["router"].set_params(z["params"], z["mean"], z["std"])
    _kept[key] = s
    return s


def _price(rng, sel):
    w = 1000.0 * min(1.0, sel)
    a = rng.uniform(0.0, 1000.0 - w)
    return And(Cmp(PRICE, ">=", a), Cmp(PRICE, "<", a + w))


def _categories(rng, n):
    return In(CATEGORY, sorted(rng.sample(range(10), max(1, min(10, n)))))


def _one_filter(rng, kind, sel):
    if kind == "range":
        return _price(rng, sel)
    if kind == "in":
        return _categories(rng, int(round(sel * 10)))
    if kind == "both":
        return And(_price(rng, sel * 5), _categories(rng, 2))
    if kind == "or":
        return And(Or(_price(rng, sel), Cmp(CATEGORY, "==", float(rng.randrange(10)))),
                   Not(Cmp(CATEGORY, "==", float(rng.randrange(10)))))
    # "each": selectivity log-uniform 0.05 %..90 %, a third with a category set
    sel = math.exp(rng.uniform(math.log(0.0005), math.log(0.9)))
    if rng.random() < 1 / 3:
        return And(_price(rng, sel * 2), _categories(rng, 5))
    return _price(rng, sel)


def _filters(rng, case):
    n, kind, sel = case["batch"], case["filter"], case["sel"]
    if kind == "none":
        return [None] * n
    if kind == "each":
        return [_one_filter(rng, kind, sel) for _ in range(n)]
    if kind == "mixed":  # the six kinds of one table's usual filters, in turn
        six = [_one_filter(rng, "both", 0.001), _price(rng, 0.01), _categories(rng, 1),
               _categories(rng, 3), _price(rng, 0.7), _price(rng, 0.95)]
        return [six[i % 6] for i in range(n)]
    return [_one_filter(rng, kind, sel)] * n


def _inputs(case, seed, centers):
    rng = random.Random(int(seed) * 7919 + 13)
    q = _mixture(_gen(int(seed) * 2 + 1), centers, case["batch"], case["values"])
    return q, _filters(rng, case), np.array([rng.choice([1, 10, 100]) for _ in range(case["batch"])],
                                            np.uint32)


def prepare(case, seed):
    if case["call"] == "build":
        centers = _centers(case["dim"], 64)
        return {"case": case, "rows": _mixture(_gen(int(seed) * 2 + 1), centers, case["rows"],
                                               case["values"])}
    s = _service(case)
    q, preds, k = _inputs(case, seed, s["centers"])
    st = {"case": case, "service": s, "q": q, "preds": preds, "k": k}
    if case["call"] in ("graph", "routed"):
        st["entries"] = s["hnsw"].entries(q)
    # a program that sends batches of one kind keeps the filters' arrays
    if case["call"] in ("brute", "routed"):
        st["filters"] = concat(preds, case["rows"], entries=st.get("entries"))
    return st


def run(state):
    case = state["case"]
    call = case["call"]
    if call == "build":
        h = Hnsw(state["rows"], case["k"], builder="gpu")
        return [h.l0, h.levels, h.upper, h.entry_node]
    s = state["service"]
    if call == "brute":
        return list(s["index"].brute_batch_raw(state["q"], state["filters"], case["k"]))
    if call == "graph":
        return list(s["index"].graph_batch(state["q"], state["entries"], state["preds"], case["k"]))
    if call == "routed":
        return list(routed_batch(s["index"], s["router"], state["q"], None, case["k"],
                                 state["entries"], topb=case["k"], bp=state["filters"])[:3])
    return list(s["stream"].run(state["q"], state["preds"], state["k"])[:3])


@functools.lru_cache(maxsize=1)
def _sample():
    rng = np.random.default_rng(5)
    return np.stack([rng.integers(0, 10, 20_000).astype(np.float64),
                     rng.uniform(0.0, 1000.0, 20_000)])


def work(case):
    n, d, b = case["rows"], case["dim"], case["batch"]
    if case["call"] == "build":
        # every row's neighbours among the rows before it: half of all pairs
        return {"bytes": n * d * 4 + n * (2 * case["k"] + 1) * 4, "flops": float(n) * n * d}
    out = b * case["k"] * 16 + b * d * 4
    if case["call"] == "graph":
        # about ef expansions of 32 neighbours, most of them met before
        seen = case["k"] * 12
        return {"bytes": b * (seen * d * 4 + case["k"] * 32 * 4) + out, "flops": 3.0 * b * seen * d}
    preds = _filters(random.Random(13), case)
    masks = [eval_numpy(p, _sample()) for p in preds]  # rows of a small table that pass
    pairs = float(sum(m.mean() for m in masks))
    union = float(np.any(masks, axis=0).mean())
    cols = 0 if case["filter"] == "none" else 1 if case["filter"] in ("range", "in") else 2
    return {"bytes": n * (union * d * ELEMENT[case["precision"]] + cols * 8) + out,
            "flops": 2.0 * n * pairs * d}


def exact(case, seed):
    """The filtered nearest neighbours by a plain 64-bit search (None: the
    call is an approximate search or returns whole numbers alone)."""
    if case["call"] in ("build", "graph"):
        return None
    s = _service(case)
    q, preds, k = _inputs(case, seed, s["centers"])
    n, b = case["rows"], case["batch"]
    kout = STREAM_K if case["call"] == "stream" else case["k"]
    qd = torch.from_numpy(q).cuda().double()
    qn = (qd * qd).sum(1)[:, None]
    best = torch.full((b, kout), math.inf, dtype=torch.float64, device="cuda")
    kinds = list({id(p): p for p in preds}.values())
    masks = torch.from_numpy(np.stack([eval_numpy(p, s["cols"]) for p in kinds]))
    which = torch.tensor([[id(x) for x in kinds].index(id(p)) for p in preds], device="cuda")
    for i in range(0, n, 1 << 18):
        x = torch.from_numpy(s["rows"][i:i + (1 << 18)]).cuda().double()
        dist = (qn + (x * x).sum(1)[None, :] - 2.0 * (qd @ x.T)).clamp_(min=0.0)
        passing = masks[:, i:i + (1 << 18)].cuda()
        dist.masked_fill_(~passing[which], math.inf)
        top = torch.topk(dist, min(kout, dist.shape[1]), dim=1, largest=False).values
        best = torch.sort(torch.cat([best, top], 1), 1).values[:, :kout]
    d = best.cpu().numpy()
    d[~np.isfinite(d)] = 0.0
    if case["call"] == "stream":
        d[np.arange(kout)[None, :] >= k[:, None]] = 0.0
    return [None, d, None, None][:3 if case["call"] in ("stream", "routed") else 4]
