"""The work users have this library do, as cases that can be timed.

A case is a plain dict. Its "kind" is the path it takes:
  flat    exact search of a FlatIndex
  ivf     an IVF fast-scan search, usually re-ranked by a RefineIndex over it
  served  a burst of mixed requests through a Server
  train   IVFIndex.train with Lloyd's k-means and the PQ codebook
  build   IVFIndex.train with the default clustering, add, and a first query
listed() names a dozen of them; draw() gives more over the same ranges.
prepare() makes the data from the seed and builds the index the way a user
does; run() is the one call (or the few calls) the user waits for.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import qann_b200 as qb

METRICS = {"l2": qb.Metric.L2, "cosine": qb.Metric.Cosine, "ip": qb.Metric.InnerProduct}


def listed():
    return [
        # An exact lookup of one vector in a collection that needs no training:
        # the smallest call there is over a table worth searching.
        _flat("flat_one_query", n=1_000_000, dim=128, nq=1, k=10, metric="l2", data="mixture"),
        # Brute-force ground truth and nearest-neighbour graphs: a large batch,
        # many results, rows of uneven length.
        _flat("flat_batch_k100", n=2_000_000, dim=96, nq=10_000, k=100, metric="l2", data="scaled", io="device"),
        # Embeddings of a text encoder (768 wide), ranked by dot product; an odd
        # number of rows and of queries, some rows deleted.
        _flat("flat_wide_ip", n=200_003, dim=768, nq=509, k=10, metric="ip", data="mixture", removed=0.01),
        # The reference's own small benchmark: 1,000 queries over 100,000 rows.
        _ivf("ivf_small_batch", n=100_000, dim=128, nlist=256, m=64, nprobe=16, k_factor=10, nq=1000, k=10,
             metric="l2", data="uniform"),
        # One interactive query against an angular index.
        _ivf("ivf_one_query", n=500_000, dim=100, nlist=2048, m=50, nprobe=64, k_factor=10, nq=1, k=10,
             metric="cosine", data="zipf"),
        # Offline batch search of the angular index at the recall users ask for,
        # queries and results on the device.
        _ivf("ivf_angular_batch", n=1_200_000, dim=100, nlist=4096, m=50, nprobe=256, k_factor=20, nq=10_000, k=10,
             metric="cosine", data="zipf", io="device"),
        # Inner product without re-ranking: an IVFIndex on its own, a rotated
        # codebook, odd sizes, deleted rows.
        _ivf("ivf_ip_ragged", n=300_007, dim=96, nlist=1000, m=48, nprobe=33, k_factor=0, nq=777, k=20, metric="ip",
             data="mixture", removed=0.02, rotate=True),
        # A where= filter evaluated to a bitmap: a tenth of the rows allowed.
        _ivf("ivf_filtered", n=500_000, dim=128, nlist=2048, m=64, nprobe=64, k_factor=10, nq=256, k=100, metric="l2",
             data="mixture", allowed=0.1, form="bitmap"),
        # A narrow allowed= list (one tenant's documents), scanned exactly.
        _ivf("ivf_narrow_filter", n=300_000, dim=128, nlist=1024, m=64, nprobe=32, k_factor=10, nq=64, k=10,
             metric="l2", data="mixture", allowed=0.015, form="ids", custom_ids=True),
        # Requests that arrive together at a server: k, nprobe and filters mixed.
        _served("served_burst", n=500_000, dim=128, nlist=4096, m=64, k_factor=10, requests=4000),
        # Training a large coarse quantizer with Lloyd iterations.
        _train("train_lloyd", n=500_000, dim=128, nlist=4096, m=64, iters=10),
        # Building an index with the default settings, and its first answers.
        _build("build_default", n=200_000, dim=100, nlist=1024, m=50, nq=100, metric="cosine"),
    ]


def _flat(name, *, n, dim, nq, k, metric, data, io="host", removed=0.0):
    return {"name": name, "kind": "flat", "n": n, "dim": dim, "nq": nq, "k": k, "metric": metric, "data": data,
            "io": io, "removed": removed}


def _ivf(name, *, n, dim, nlist, m, nprobe, k_factor, nq, k, metric, data, io="host", removed=0.0, rotate=False,
         allowed=0.0, form="none", custom_ids=False):
    return {"name": name, "kind": "ivf", "n": n, "dim": dim, "nlist": nlist, "m": m, "nprobe": nprobe,
            "k_factor": k_factor, "nq": nq, "k": k, "metric": metric, "data": data, "io": io, "removed": removed,
            "rotate": rotate, "allowed": allowed, "form": form, "custom_ids": custom_ids}


def _served(name, *, n, dim, nlist, m, k_factor, requests):
    return {"name": name, "kind": "served", "n": n, "dim": dim, "nlist": nlist, "m": m, "k_factor": k_factor,
            "nq": requests, "metric": "l2", "data": "mixture"}


def _train(name, *, n, dim, nlist, m, iters):
    return {"name": name, "kind": "train", "n": n, "dim": dim, "nlist": nlist, "m": m, "iters": iters, "metric": "l2",
            "data": "mixture"}


def _build(name, *, n, dim, nlist, m, nq, metric):
    return {"name": name, "kind": "build", "n": n, "dim": dim, "nlist": nlist, "m": m, "nq": nq, "k": 10,
            "nprobe": max(1, nlist // 32), "metric": metric, "data": "zipf"}


def _log(rng, lo, hi):
    """A whole number spread evenly over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dim_m(rng, widest):
    """A dimension, odd multiples among them, and sub-quantizers that divide it."""
    sd = rng.choice([2, 2, 2, 3, 4])
    m = 2 * rng.randint(4, widest // sd // 2)   # (fast-scan codes come in pairs)
    return m * sd, m


def draw(rng):
    kind = rng.choice(["flat", "flat", "ivf", "ivf", "ivf", "ivf", "served", "train", "build"])
    metric = rng.choice(["l2", "l2", "cosine", "ip"])
    if kind == "flat":
        nq = _log(rng, 1, 10_000)
        dim = rng.choice([rng.randint(16, 128), rng.randint(16, 128), rng.randint(129, 768)])
        rows = min(2_000_000, int(200_000_000 / dim), int(1.8e12 / (nq * dim * max(1, dim // 96))))
        return {k: v for k, v in _flat("", n=_log(rng, 1000, max(1001, rows)), dim=dim, nq=nq, k=_log(rng, 1, 100),
                                       metric=metric, data=rng.choice(["mixture", "scaled", "uniform"]),
                                       io=rng.choice(["host", "device"]),
                                       removed=rng.choice([0.0, 0.0, 0.05])).items() if k != "name"}
    n = _log(rng, 30_000, 600_000)
    nlist = max(100, int(n / rng.uniform(100, 400)))
    if kind == "ivf":
        dim, m = _dim_m(rng, rng.choice([128, 128, 256]))
        form = rng.choice(["none", "none", "none", "ids", "bitmap"])
        io = rng.choice(["host", "device"]) if form == "none" else "host"
        k = _log(rng, 1, 100)
        nq = _log(rng, 1, 4000 if form == "none" else 500)
        # (a filter that no RefineIndex would answer by a direct scan, or a narrow one)
        allowed = 0.0 if form == "none" else rng.choice([rng.uniform(0.002, 0.02), rng.uniform(0.08, 0.5)])
        return {k: v for k, v in _ivf("", n=n, dim=dim, nlist=nlist, m=m, nprobe=min(nlist, _log(rng, 4, 256)),
                                      k_factor=rng.choice([0, 5, 10, 20]), nq=nq, k=k, metric=metric,
                                      data=rng.choice(["mixture", "zipf", "uniform"]), io=io,
                                      removed=rng.choice([0.0, 0.0, 0.03]), rotate=rng.random() < 0.2,
                                      allowed=allowed, form=form, custom_ids=rng.random() < 0.3).items()
                if k != "name"}
    dim, m = _dim_m(rng, 128)
    if kind == "served":
        case = _served("", n=n, dim=dim, nlist=nlist, m=m, k_factor=10, requests=_log(rng, 200, 4000))
    elif kind == "train":
        nlist = min(16_384, max(100, int(n / rng.uniform(30, 400))))
        case = _train("", n=n, dim=dim, nlist=nlist, m=m, iters=max(1, min(rng.randint(2, 10), int(1.9e10 / n / nlist))))
    else:
        n = min(n, 200_000)
        case = _build("", n=n, dim=dim, nlist=max(100, n // 200), m=m, nq=_log(rng, 1, 200), metric=metric)
    return {k: v for k, v in case.items() if k != "name"}


# ---- inputs ---------------------------------------------------------------------


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _vectors(case, seed, count, part):
    """`count` rows of the case's distribution on the GPU, float32. The rows
    (part 0) and the queries (part 1) share the mixture's centres."""
    dim, data = case["dim"], case["data"]
    g = _gen(3 * seed + 1 + part)
    if data == "uniform":
        return torch.rand(count, dim, generator=g, device="cuda")
    x = torch.randn(count, dim, generator=g, device="cuda")
    if data == "scaled":   # unequal row lengths: LogNormal(0, 0.25)
        return x.mul_(torch.exp(0.25 * torch.randn(count, 1, generator=g, device="cuda")))
    centres = torch.randn(2000, dim, generator=_gen(3 * seed + 3), device="cuda")
    if data == "zipf":     # cluster sizes by Zipf(1.1), sigma 0.3
        p = torch.arange(1, 2001, device="cuda", dtype=torch.float64) ** -1.1
        edges = torch.cumsum(p / p.sum(), 0)
        u = torch.rand(count, generator=g, device="cuda", dtype=torch.float64)
        lab = torch.searchsorted(edges, u).clamp_(max=1999)
        return x.mul_(0.3).add_(centres[lab])
    lab = torch.randint(0, 2000, (count,), generator=g, device="cuda")
    return x.mul_(0.2).add_(centres[lab])


def _removed_rows(case, seed):
    count = int(case.get("removed", 0.0) * case["n"])
    return np.random.default_rng(seed + 77).choice(case["n"], count, replace=False) if count else None


def _label(case, rows):
    """The ids the rows are known by."""
    return rows * 7 + 3 if case.get("custom_ids") else rows


def _allowed_rows(case, seed):
    count = max(1, int(case["allowed"] * case["n"]))
    return np.sort(np.random.default_rng(seed + 99).choice(case["n"], count, replace=False))


def _train_sample(rows, nlist):
    """What is trained on: a sample of the rows, as collections of this size are."""
    return rows[:max(40 * nlist, 20_000)]


def _index(case, seed, rows):
    """The index a search case searches, trained and filled."""
    n, custom = case["n"], bool(case.get("custom_ids"))
    ids = _label(case, np.arange(n, dtype=np.int64)) if custom else None
    if case["kind"] == "flat":
        index = qb.FlatIndex(case["dim"], metric=METRICS[case["metric"]])
        index.add(rows)
    else:
        refine = case["k_factor"] > 0
        ivf = qb.IVFIndex(case["dim"], case["nlist"], case.get("nprobe", 16), metric=METRICS[case["metric"]],
                          custom_ids=custom and not refine)
        ivf.enable_pq(case["m"], fast_scan=True, rotate=bool(case.get("rotate")))
        ivf.train(_train_sample(rows, case["nlist"]), max_iters=4, seed=1, clustering=qb.Clustering.Lloyd)
        index = qb.RefineIndex(ivf, case["k_factor"], custom_ids=custom) if refine else ivf
        index.add(rows, ids)
    gone = _removed_rows(case, seed)
    if gone is not None:
        index.remove(_label(case, gone))
    return index


def prepare(case, seed):
    kind = case["kind"]
    rows_dev = _vectors(case, seed, case["n"], 0)
    rows = rows_dev.cpu().numpy()
    del rows_dev
    if kind == "train":
        return {"case": case, "rows": rows}
    queries = _vectors(case, seed, case["nq"], 1)
    state = {"case": case, "q": queries.cpu().numpy()}
    if kind == "build":
        state["rows"] = rows
        return state
    index = _index(case, seed, rows)
    state["index"] = index
    if kind == "served":
        state.update(_requests(case, seed, index))
        return state
    if case["io"] == "device":
        state["q_dev"] = queries
        state["ids"] = torch.empty(case["nq"], case["k"], dtype=torch.int64, device="cuda")
        state["d"] = torch.empty(case["nq"], case["k"], dtype=torch.float32, device="cuda")
    if case.get("form") == "ids":
        state["allowed"] = _label(case, _allowed_rows(case, seed)).astype(np.int64)
    elif case.get("form") == "bitmap":
        state["words"] = _bitmap(case["n"], _allowed_rows(case, seed))
    index.batch_query(state["q"][:1], case["k"])   # the index goes to the GPU before the first request
    return state


def _bitmap(n, rows):
    bits = np.zeros((n + 63) // 64 * 64, np.uint8)
    bits[rows] = 1
    return np.packbits(bits, bitorder="little").view(np.uint64)


def _requests(case, seed, index):
    """k of 10 or 100, nprobe log-uniform in 8..256, three in ten filtered by
    one of eight bitmaps of 5 % to 50 %; all waiting when the pass begins."""
    rng = np.random.default_rng(seed + 5)
    nq, n = case["nq"], case["n"]
    server = qb.Server(index, slots=2, max_batch=512)
    filters = [server.add_filter(_bitmap(n, np.nonzero(rng.random(n) < s)[0])) for s in rng.uniform(0.05, 0.5, 8)]
    pick = np.where(rng.random(nq) < 0.3, rng.choice(filters, nq), -1)
    return {"server": server, "ks": rng.choice([10, 100], nq).astype(np.int32),
            "nprobes": np.minimum(case["nlist"], np.exp(rng.uniform(np.log(8), np.log(256), nq))).astype(np.int32),
            "filters": pick.astype(np.int32), "arrivals": np.zeros(nq)}


# ---- the passes -----------------------------------------------------------------


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "train":
        ivf = qb.IVFIndex(case["dim"], case["nlist"])
        ivf.enable_pq(case["m"], fast_scan=True)
        ivf.train(state["rows"], max_iters=case["iters"], seed=1, clustering=qb.Clustering.Lloyd)
        return {"centroids": ivf.centroids()}
    if kind == "build":
        ivf = qb.IVFIndex(case["dim"], case["nlist"], case["nprobe"], metric=METRICS[case["metric"]])
        ivf.enable_pq(case["m"], fast_scan=True)
        ivf.train(state["rows"], seed=1)
        index = qb.RefineIndex(ivf, 10)
        added = index.add(state["rows"])
        ids, d = index.batch_query(state["q"], case["k"])
        return {"centroids": ivf.centroids(), "sizes": ivf.list_sizes().astype(np.int64), "added": added, "ids": ids,
                "d": d}
    if kind == "served":
        ids, d, _ = state["server"].replay(state["q"], state["ks"], state["arrivals"], nprobes=state["nprobes"],
                                           filter_ids=state["filters"])
        return {"ids": ids, "d": d}
    index = state["index"]
    if case["io"] == "device":
        index.search_device(state["q_dev"].data_ptr(), case["nq"], case["k"], state["ids"].data_ptr(),
                            state["d"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return {"ids": state["ids"], "d": state["d"]}
    if "words" in state:
        ids, d = index.batch_query_bitmap(state["q"], case["k"], state["words"])
    else:
        ids, d = index.batch_query(state["q"], case["k"], allowed=state.get("allowed"))
    return {"ids": ids, "d": d}


def work(case):
    """Each input once, each output once; multiply-adds count two. An IVF
    search cannot do without the codes of the lists that are probed at least
    once, the coarse products and one addition per code it scans."""
    n, dim, nq = case["n"], case["dim"], case.get("nq", 0)
    kind = case["kind"]
    if kind == "flat":
        return {"bytes": 4 * n * dim + 4 * nq * dim + 12 * nq * case["k"], "flops": 2 * nq * n * dim}
    nlist, m = case["nlist"], case["m"]
    tables = 4 * nlist * dim + 64 * dim
    train = 0
    if kind in ("train", "build"):
        # the rows against the centroids once an iteration (or pass) and once more, 25 iterations of the codebook
        rounds = case.get("iters", 2) + 1
        train = 2 * rounds * n * nlist * dim + 26 * 2 * min(n, 4096) * 16 * dim
    if kind == "train":
        return {"bytes": 4 * n * dim + tables, "flops": train}
    k = case.get("k", 55)
    nprobe = min(nlist, case.get("nprobe", 72))
    if case.get("form", "none") != "none" and case["k_factor"] and int(case["allowed"] * n) <= 6 * nlist:
        rows = int(case["allowed"] * n)   # a RefineIndex scores a narrow filter's rows exactly
        return {"bytes": 4 * rows * dim + 8 * rows + 4 * nq * dim + 12 * nq * k, "flops": 2 * nq * rows * dim}
    touched = 1.0 - (1.0 - nprobe / nlist) ** nq
    kp = k * case.get("k_factor", 10)
    codes = int(n * (m / 2 + 4) * touched)
    rows = 4 * dim * min(n, nq * kp)
    out = {"bytes": tables + codes + rows + 4 * nq * dim + 12 * nq * k,
           "flops": 2 * nq * nlist * dim + int(nq * (nprobe / nlist) * n * m) + 2 * nq * kp * dim}
    if case.get("form", "none") != "none":
        out["bytes"] += n // 8
    if kind == "build":
        out["bytes"] += 8 * n * dim
        out["flops"] += train
    return out


def exact(case, seed):
    """The exact distances where the answer is exact by definition: flat
    searches, and a RefineIndex's scan of a narrow filter's rows. The
    candidates of a fast-scan and the steps of a clustering have no value
    apart from the arithmetic that makes them, and ids are whole numbers."""
    narrow = (case["kind"] == "ivf" and case["form"] != "none" and case["k_factor"] > 0 and
              len(_allowed_rows(case, seed)) <= 6 * case["nlist"])
    if case["kind"] != "flat" and not narrow:
        return None
    x = _vectors(case, seed, case["n"], 0)
    live = torch.ones(case["n"], dtype=torch.bool, device="cuda")
    gone = _removed_rows(case, seed)
    if gone is not None:
        live[torch.from_numpy(gone).cuda()] = False
    if narrow:
        allowed = torch.zeros_like(live)
        allowed[torch.from_numpy(_allowed_rows(case, seed)).cuda()] = True
        live &= allowed
        if not 0 < int(live.sum()) <= 6 * case["nlist"]:
            return None
    x = x[live]
    k, q = case["k"], _vectors(case, seed, case["nq"], 1).double()
    if case["metric"] == "cosine":
        q = q / q.norm(dim=1, keepdim=True)
    best = torch.full((case["nq"], k), math.inf, dtype=torch.float64, device="cuda")
    step = max(1000, int(4e8 / max(1, case["nq"])))
    for r0 in range(0, x.shape[0], step):
        b = x[r0:r0 + step].double()
        if case["metric"] == "cosine":
            b = b / b.norm(dim=1, keepdim=True)
        s = q @ b.T
        if case["metric"] == "l2":
            s = (q * q).sum(1, keepdim=True) + (b * b).sum(1)[None] - 2 * s
        else:
            s = 1 - s if case["metric"] == "cosine" else -s
        s = torch.topk(s, min(k, s.shape[1]), dim=1, largest=False).values
        best = torch.topk(torch.cat([best, s], 1), k, dim=1, largest=False).values
    return {"ids": None, "d": best.cpu() if case["io"] == "host" else best}
