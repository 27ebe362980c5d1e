"""The calls a graph-learning program makes of this framework, as cases that can be timed.

A training or serving step samples a mini-batch (``sample_minibatch``, or hop by hop with
``csr_sampling`` / ``csr_cache_sampling`` and ``tensor_relabel``), fetches the frontier's feature
rows from a table that is cached on the GPU in whole or in part (``cache_fetch`` and its mask form)
and, where rows are trained, writes them back (``cache_set``).  Between steps the cache is refilled
(``cache_insert_set``), ids are relabelled and degree arrays are scanned into row offsets.

Sizes come from the benchmark's workloads (2,400,000 nodes / 62,000,000 edges, 2,400,000 x 100
float32 rows, batches of 500,000 ids, fan-outs 15/10/5, 4,000,000 keys of 256 bfloat16, scans and
relabels beyond the L2 cache) and from the small and odd ends of the same ranges.
"""
import math

import numpy as np
import torch

from shmtensor_b200 import capi

_DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16, "float16": torch.float16,
           "int32": torch.int32, "int64": torch.int64}
_ITEM = {"float32": 4, "bfloat16": 2, "float16": 2, "int32": 4, "int64": 8}
_ZIPF, _UNIFORM_SHARE = 1.1, 0.21  # popularity of rows in a batch, and its part without a bias
_DEG_TAIL, _DEG_CAP = 1.1, 10_000  # node degrees: P(deg > d) ~ d^-1.1, at most 10,000


def listed():
    return [
        # one hop for a handful of requested nodes, through the per-hop calls: latency and launches
        {"name": "hop_small", "kind": "hop", "nodes": 100_000, "degree": 20.0, "on": "gpu", "cached": 0.0,
         "ids": "int64", "seeds": 100, "fanout": 10, "replace": False},
        # the training step's sampler on a graph in pinned host memory, hot fifth of the nodes cached
        {"name": "minibatch_host", "kind": "minibatch", "nodes": 2_400_000, "degree": 25.8, "on": "host", "cached": 0.2,
         "ids": "int32", "seeds": 1024, "fanouts": "5,10,15", "replace": False, "option": "plain"},
        # large batches on a graph that fits the GPU's memory, with edge ids (edge features follow)
        {"name": "minibatch_gpu_large", "kind": "minibatch", "nodes": 10_000_000, "degree": 20.0, "on": "gpu", "cached": 0.0,
         "ids": "int64", "seeds": 8192, "fanouts": "5,10,15", "replace": False, "option": "eids"},
        # importance sampling: neighbours picked in proportion to edge weights
        {"name": "minibatch_weighted", "kind": "minibatch", "nodes": 2_400_000, "degree": 25.8, "on": "gpu", "cached": 0.0,
         "ids": "int32", "seeds": 1000, "fanouts": "10,15", "replace": False, "option": "weighted"},
        # feature rows of one serving request
        {"name": "fetch_small", "kind": "fetch", "rows": 100_000, "dim": 128, "dtype": "float32", "on": "host", "cached": 0.2,
         "ids": "int64", "n": 100, "mask": False},
        # the benchmark's batch: table in pinned host memory, a fifth of the rows cached, four of five ids hit
        {"name": "fetch_mixed", "kind": "fetch", "rows": 2_400_000, "dim": 100, "dtype": "float32", "on": "host", "cached": 0.2,
         "ids": "int64", "n": 500_000, "mask": False},
        # a table that is cached whole, a large frontier
        {"name": "fetch_resident", "kind": "fetch", "rows": 4_000_000, "dim": 100, "dtype": "float32", "on": "gpu", "cached": 1.0,
         "ids": "int64", "n": 1_200_000, "mask": False},
        # odd-width half-precision rows (602 bytes), slots looked up once and used as a mask
        {"name": "fetch_ragged", "kind": "fetch", "rows": 1_000_000, "dim": 301, "dtype": "bfloat16", "on": "gpu", "cached": 1.0,
         "ids": "int32", "n": 150_001, "mask": True},
        # writing trained rows back: hits overwrite the cached row, the others the host table
        {"name": "set_mixed", "kind": "set", "rows": 500_000, "dim": 100, "dtype": "float32", "on": "host", "cached": 0.9,
         "ids": "int64", "n": 200_003},
        # filling an empty cache and looking ids up in it, half of them absent
        {"name": "cache_fill", "kind": "fill", "keys": 4_000_000, "dim": 256, "dtype": "bfloat16", "ids": "int64",
         "lookups": 1_000_000},
        # renumbering the ids of a partition: far more ids than the L2 cache holds
        {"name": "relabel_large", "kind": "relabel", "n": 33_554_432, "distinct": 0.125, "sparse": True, "ids": "int64",
         "parts": 1},
        # degrees of a graph's nodes to row offsets
        {"name": "scan_degrees", "kind": "scan", "n": 2_400_001, "ids": "int64", "exclusive": True},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm; odd ones among them."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["hop", "minibatch", "minibatch", "weighted", "fetch", "fetch", "fetch", "mask", "set", "fill",
                       "relabel", "scan"])
    ids = rng.choice(["int32", "int64"])
    if kind in ("hop", "minibatch", "weighted"):
        on = rng.choice(["gpu", "host"]) if kind != "weighted" else "gpu"
        case = {"kind": "hop" if kind == "hop" else "minibatch", "nodes": _log(rng, 50_000, 2_400_000 if on == "host" else 10_000_000),
                "degree": round(rng.uniform(6.0, 25.0), 1), "on": on, "cached": 0.0 if on == "gpu" else rng.choice([0.0, 0.2, 0.5]),
                "ids": ids}
        if kind == "hop":
            case.update(seeds=_log(rng, 50, 60_000 if on == "gpu" else 8_000), fanout=rng.choice([3, 5, 10, 15, 25, 40]),
                        replace=rng.random() < 0.25)
        elif kind == "weighted":
            case.update(seeds=_log(rng, 50, 1000), fanouts=rng.choice(["5,10", "10,15", "10,5", "20"]), replace=False,
                        option="weighted")
        else:
            case.update(seeds=_log(rng, 50, 8192 if on == "gpu" else 1024), fanouts=rng.choice(["5,10,15", "10,10", "10,25", "5,5,5"]),
                        replace=rng.random() < 0.25, option=rng.choice(["plain", "plain", "eids"]))
        return case
    if kind in ("fetch", "mask", "set"):
        dtype = rng.choice(["float32", "bfloat16", "float16"])
        dim = rng.choice([32, 64, 100, 128, 256, rng.randrange(17, 602)])
        row = dim * _ITEM[dtype]
        on = rng.choice(["gpu", "gpu", "host"])
        rows = _log(rng, 50_000, min(4_000_000, (1600 if on == "gpu" else 400) * 1_000_000 // row))
        top = min(500_000_000 // row, 1_200_000) if on == "gpu" else min(100_000_000 // row, 300_000)
        case = {"kind": "set" if kind == "set" else "fetch", "rows": rows, "dim": dim, "dtype": dtype, "on": on,
                "cached": 1.0 if on == "gpu" else rng.choice([0.2, 0.5, 0.9]), "ids": ids,
                "n": _log(rng, 64, min(top, rows // 2 if kind == "set" else top))}
        if kind != "set":
            case["mask"] = kind == "mask"
        return case
    if kind == "fill":
        dtype = rng.choice(["float32", "bfloat16"])
        dim = rng.choice([64, 100, 128, 256])
        keys = _log(rng, 5_000, 2_000_000_000 // max(512, dim * _ITEM[dtype]))
        return {"kind": "fill", "keys": keys, "dim": dim, "dtype": dtype, "ids": ids, "lookups": max(100, keys // 4)}
    if kind == "relabel":
        return {"kind": "relabel", "n": _log(rng, 1_000, 16_000_000), "distinct": rng.choice([0.1, 0.3, 0.8]),
                "sparse": ids == "int64" and rng.random() < 0.5, "ids": ids, "parts": rng.choice([1, 2, 3])}
    return {"kind": "scan", "n": _log(rng, 1_000, 110_000_000), "ids": ids, "exclusive": rng.random() < 0.5}


# --------------------------------------------------------------------------- inputs
def _host_copy(t):
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    out.copy_(t)
    return out


def _degrees_at(u, degree):
    """Degrees of nodes at quantiles ``u`` in (0, 1], scaled to the wanted mean, and the fraction
    behind the whole part (numpy and torch)."""
    q = (np.arange(20_000) + 0.5) / 20_000
    raw = np.minimum(np.floor(q ** (-1.0 / _DEG_TAIL)), _DEG_CAP)
    scale = degree / raw.mean()
    lib = np if isinstance(u, np.ndarray) else torch
    d = lib.floor(u ** (-1.0 / _DEG_TAIL)).clip(0, _DEG_CAP) * scale
    return d.clip(0, _DEG_CAP)


def _graph(case, g):
    """Power-law CSR on the GPU; a row's neighbours are an arithmetic progression modulo the node
    count (distinct, spread over the nodes).  The shape of the graph is the case's; which node has
    which number, and so where every row lies, comes from ``g``: a sample of the same stream of
    draws has the same sizes whatever the numbering."""
    n, dev = case["nodes"], "cuda"
    fixed = torch.Generator(device=dev).manual_seed(3)
    u = torch.rand(n, generator=fixed, device=dev, dtype=torch.float64).clip(min=1e-9)
    deg = (_degrees_at(u, case["degree"]) + torch.rand(n, generator=fixed, device=dev)).long()
    primes = torch.tensor([7, 11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47, 53, 59, 61, 67], device=dev)
    base = torch.randint(0, n, (n,), generator=fixed, device=dev)
    step = primes[torch.randint(0, 16, (n,), generator=fixed, device=dev)]
    seeds = torch.randperm(n, generator=fixed, device=dev)[:case["seeds"]]
    node_at = torch.randperm(n, generator=g, device=dev)  # numbering: node at each number ...
    number = torch.empty_like(node_at)                    # ... and number of each node
    number[node_at] = torch.arange(n, device=dev)
    deg = deg[node_at]
    indptr = torch.zeros(n + 1, dtype=torch.int64, device=dev)
    torch.cumsum(deg, 0, out=indptr[1:])
    total = int(indptr[-1])
    indices = torch.empty(total, dtype=_DTYPES[case["ids"]], device=dev)
    weights = torch.empty(total, device=dev) if case.get("option") == "weighted" else None
    for lo in range(0, n, 2_000_000):
        hi = min(n, lo + 2_000_000)
        a, b = int(indptr[lo]), int(indptr[hi])
        at = torch.repeat_interleave(torch.arange(lo, hi, device=dev), deg[lo:hi], output_size=b - a)
        j = torch.arange(a, b, device=dev) - indptr[at]
        row = node_at[at]
        indices[a:b] = number[(base[row] + j * step[row]) % n].to(indices.dtype)
        if weights is not None:  # a float in (0.05, 1.05) of (node, position)
            x = row * 0x9E3779B97F4A7C1 + j * 0x2545F4914F6CDD1D
            x = (x ^ (x >> 29)) * 0x94D049BB133111E
            weights[a:b] = ((x >> 24) & 0xFFFFF) / float(1 << 20) + 0.05
    return indptr, indices, deg, number[seeds].to(indices.dtype), weights


def _graph_state(case, g):
    indptr, indices, deg, seeds, weights = _graph(case, g)
    s = {"seeds": seeds, "weights": weights, "cached": {}}
    if case["on"] == "host":
        s["indptr"], s["indices"] = _host_copy(indptr), _host_copy(indices)
        if case["cached"] > 0:
            hot = torch.argsort(deg, descending=True, stable=True)[:int(case["nodes"] * case["cached"])]
            gp, gi = capi.create_subcsr(s["indptr"], s["indices"], hot)
            slots = torch.arange(hot.numel(), dtype=torch.int32, device="cuda")
            s["cached"] = {"gpu_indptr": gp, "gpu_indices": gi, "hashmap": capi.CUCOStaticHashmap(hot.int(), slots, 0.8)}
            if case.get("option") == "eids":
                s["cached"]["gpu_edge_base"] = capi.subcsr_edge_base(s["indptr"], hot)
    else:
        s["indptr"], s["indices"] = indptr, indices
    return s


def _row_values(n, case, g):
    """``n`` feature rows on the GPU."""
    out = torch.empty(n, case["dim"], dtype=_DTYPES[case["dtype"]], device="cuda")
    for lo in range(0, n, 500_000):
        hi = min(n, lo + 500_000)
        out[lo:hi] = torch.randn(hi - lo, case["dim"], generator=g, device="cuda")
    return out


def _popularity(rows):
    w = torch.arange(1, rows + 1, device="cuda", dtype=torch.float64) ** -_ZIPF
    return torch.cumsum(w, 0) / w.sum()


def _table_state(case, g):
    rows, n = case["rows"], case["n"]
    ranking = torch.randperm(rows, generator=g, device="cuda")  # rows by popularity
    table = _row_values(rows, case, g)
    n_hot = int(rows * case["cached"])
    hot = ranking[:n_hot]
    s = {"uva": _host_copy(table) if case["on"] == "host" else None, "gpu": table[hot]}
    key_dtype = _DTYPES[case["ids"]]
    s["map"] = capi.CUCOStaticHashmap(hot.to(key_dtype), torch.arange(n_hot, dtype=torch.int32, device="cuda"), 0.5)
    if case["kind"] == "set":  # the distinct rows of a step, once each
        ids = torch.randperm(rows, generator=g, device="cuda")[:n]
        s["update"] = _row_values(n, case, g)
    else:
        n_flat = int(n * _UNIFORM_SHARE)
        rank = torch.searchsorted(_popularity(rows), torch.rand(n - n_flat, generator=g, device="cuda", dtype=torch.float64))
        ids = torch.cat([ranking[rank.clip(max=rows - 1)], torch.randint(0, rows, (n_flat,), generator=g, device="cuda")])
        ids = ids[torch.randperm(n, generator=g, device="cuda")]
    s["ids"] = ids.to(key_dtype)
    return s


def _distinct_ids(n, dtype, g, top):
    """``n`` distinct keys below ``top``, in random order."""
    got = torch.randint(0, top, (n + n // 16 + 1000,), generator=g, device="cuda").unique()
    return got[torch.randperm(got.numel(), generator=g, device="cuda")[:n]].to(dtype)


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    kind = case["kind"]
    if kind in ("hop", "minibatch"):
        s = _graph_state(case, g)
        if kind == "minibatch":
            s["fanouts"] = [int(k) for k in case["fanouts"].split(",")]
    elif kind in ("fetch", "set"):
        s = _table_state(case, g)
    elif kind == "fill":
        half = case["lookups"] // 2
        top = 1 << (40 if case["ids"] == "int64" else 30)
        keys = _distinct_ids(case["keys"], _DTYPES[case["ids"]], g, top)
        present = keys[torch.randint(0, keys.numel(), (half,), generator=g, device="cuda")]
        absent = torch.randint(top, 2 * top - 1, (case["lookups"] - half,), generator=g, device="cuda").to(keys.dtype)
        req = torch.cat([present, absent])
        s = {"keys": keys, "requests": req[torch.randperm(req.numel(), generator=g, device="cuda")],
             "slots": torch.arange(keys.numel(), dtype=torch.int32, device="cuda"), "rows": _row_values(keys.numel(), case, g),
             "gpu": torch.zeros(keys.numel(), case["dim"], dtype=_DTYPES[case["dtype"]], device="cuda")}
    elif kind == "relabel":
        n_ids = max(1, int(case["n"] * case["distinct"]))
        fixed = torch.Generator(device="cuda").manual_seed(4)  # which elements are equal: the case's, so is their number
        which = torch.randint(0, n_ids, (case["n"],), generator=fixed, device="cuda")
        ids = (_distinct_ids(n_ids, torch.int64, g, 1 << 43) if case["sparse"] else
               torch.randperm(n_ids, generator=g, device="cuda"))[which]
        s = {"parts": [p.clone() for p in ids.to(_DTYPES[case["ids"]]).chunk(case["parts"])]}
    else:
        s = {"data": torch.randint(0, 50, (case["n"],), generator=g, device="cuda", dtype=_DTYPES[case["ids"]])}
    s["case"] = case
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "hop":
        capi.set_sampling_seed(7777)
        c = state["cached"]
        if c:
            indptr, indices = capi.csr_cache_sampling(state["indptr"], state["indices"], c["gpu_indptr"], c["gpu_indices"],
                                                      c["hashmap"], state["seeds"], case["fanout"], case["replace"])
        else:
            indptr, indices = capi.csr_sampling(state["indptr"], state["indices"], state["seeds"], case["fanout"], case["replace"])
        frontier, local = capi.tensor_relabel([state["seeds"], indices])
        return [indptr, indices, frontier, *local]
    if kind == "minibatch":
        capi.set_sampling_seed(7777)
        extra = {"weights": state["weights"]} if case["option"] == "weighted" else {"return_eids": case["option"] == "eids"}
        frontier, hops = capi.sample_minibatch(state["indptr"], state["indices"], state["seeds"], state["fanouts"],
                                               case["replace"], **state["cached"], **extra)
        return [frontier, [list(h) for h in hops]]
    if kind == "fetch":
        if case["mask"]:
            mask = state["map"].query(state["ids"])
            return [mask, capi.cache_fetch_with_mask(state["uva"], state["gpu"], state["ids"], mask)]
        return capi.cache_fetch(state["uva"], state["gpu"], state["ids"], state["map"])
    if kind == "set":
        capi.cache_set(state["uva"], state["gpu"], state["ids"], state["update"], state["map"])
        return [state["gpu"]] if state["uva"] is None else [state["gpu"], state["uva"]]
    if kind == "fill":
        m = capi.CUCOStaticHashmap.empty(2 * state["keys"].numel(), state["keys"].dtype, torch.int32)
        capi.cache_insert_set(state["gpu"], state["keys"], state["slots"], state["rows"], m)
        return [state["gpu"], m.query(state["requests"])]
    if kind == "relabel":
        unique, local = capi.tensor_relabel(state["parts"])
        return [unique, *local]
    if case["exclusive"]:
        capi.exclusive_scan_(state["data"])
    else:
        capi.thrust_scan(state["data"])
    return state["data"]


# --------------------------------------------------------------------------- what a pass cannot do without
def _distinct(n, population):
    return population * -math.expm1(-n / population)


def work(case):
    kind = case["kind"]
    if kind in ("hop", "minibatch"):
        item = _ITEM[case["ids"]]
        q = (np.arange(20_000) + 0.5) / 20_000
        deg = _degrees_at(q, case["degree"])
        moved, n = 0.0, float(case["seeds"])
        for k in [case["fanout"]] if kind == "hop" else [int(x) for x in case["fanouts"].split(",")]:
            edges = n * float(np.where(deg > 0.5, k, 0).mean() if case["replace"] else np.minimum(deg, k).mean())
            after = n + _distinct(edges, case["nodes"])
            # ids and bounds in, offsets out; neighbours in and out, relabelled; the frontier out
            moved += n * (item + 16 + 8) + edges * 2 * item + (n + edges) * item + after * item
            if case["cached"] > 0:
                moved += n * 16
            if case.get("option") == "eids":
                moved += edges * 8
            if case.get("option") == "weighted":
                moved += n * float(deg.mean()) * 4
            n = after
        return {"bytes": moved, "flops": 0.0}
    if kind in ("fetch", "set"):
        row, n, rows = case["dim"] * _ITEM[case["dtype"]], case["n"], case["rows"]
        probe = 16 + (8 if case.get("mask") else 0)
        if kind == "set":
            read = n
        else:
            n_flat = n * _UNIFORM_SHARE
            w = np.arange(1, rows + 1, dtype=np.float64) ** -_ZIPF
            p = w / w.sum() * (n - n_flat) + n_flat / rows
            read = float(-np.expm1(-p).sum())
        return {"bytes": n * (_ITEM[case["ids"]] + probe) + (read + n) * row, "flops": 0.0}
    if kind == "fill":
        row, n = case["dim"] * _ITEM[case["dtype"]], case["keys"]
        # the empty table is written, every key claims a slot of it; a lookup reads one
        return {"bytes": n * (_ITEM[case["ids"]] + 4 + 32 + 16 + 2 * row) + case["lookups"] * (_ITEM[case["ids"]] + 16 + 4),
                "flops": 0.0}
    if kind == "relabel":
        item = _ITEM[case["ids"]]
        return {"bytes": case["n"] * (2 * item) + _distinct(case["n"], max(1, case["n"] * case["distinct"])) * item, "flops": 0.0}
    return {"bytes": case["n"] * 2 * _ITEM[case["ids"]], "flops": 0.0}


def tolerance(case):
    """Rows are moved as bytes; ids, offsets and picks (of a pinned random stream) are whole numbers."""
    return "exact"
