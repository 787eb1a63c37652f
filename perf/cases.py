"""The calls that programs make of this package, as cases that can be timed and compared: what one case works on
(`prepare`), the call itself (`run`), what it cannot do without (`work`), and how far a correct answer may lie from
another (`tolerance`). `listed` names the cases, `draw` gives more of the same ranges.

Seven paths, all through the public Python calls:
  search     `Index.search` on an index that is built once: the plain call, with one mask for all queries ("bitset") or
             one mask per query ("bitmap")
  labels     `Index.search(labels=...)` on a labelled index that has seen removals and additions
  keys       `KeyCache.topk`: the keys every query of a decoding batch attends to
  decode     `KeyCache.append` of one new key per head, then `KeyCache.topk`: a decoding step
  select     `flashinfer.ExactTopK.select` over sequences of different lengths
  prefill    `topk`: the keys of a prompt go into a new cache, which is asked
  one_call   `search`: an index is built from the vectors, asked and given up again
"""

import math
import random

import torch

import libcertex_b200 as certex
from libcertex_b200 import flashinfer, synthetic

_DTYPES = {"float32": torch.float32, "float16": torch.float16, "int8": torch.int8, "uint8": torch.uint8}
_BYTES = {"float32": 4, "float16": 2, "int8": 1, "uint8": 1}
_STEPS = 512  # decoding steps whose keys are at hand; the sequence of keys starts again after them


def _search(name, dtype, metric, n, dim, queries, k, filter="none", batch=2048):
    return {"name": name, "path": "search", "dtype": dtype, "metric": metric, "n": n, "dim": dim, "queries": queries, "k": k,
            "filter": filter, "batch": batch}


def _cache(name, path, keys, k, rows, kv_heads=8, heads=32, dim=128):
    return {"name": name, "path": path, "kv_heads": kv_heads, "heads": heads, "dim": dim, "keys": keys, "rows": rows, "k": k}


def listed():
    return [
        # one question to a small collection, as an application asks it while somebody waits: latency and launches only
        _search("one_query_3k_f32", "float32", "l2", 3000, 128, 1, 10),
        # the same to a collection of ordinary size: one pass over the codes
        _search("one_query_1m_u8", "uint8", "l2", 1_000_000, 128, 1, 10),
        # an ordinary batch over an ordinary collection (the correctness configuration of the benchmark set)
        _search("batch_100k_f32", "float32", "l2", 100_000, 128, 1000, 10),
        # sizes that fill no tile, signed bytes, the inner product, one mask for all queries (search within a subset)
        _search("masked_ragged_i8", "int8", "ip", 1_234_567, 100, 777, 33, filter="bitset"),
        # the headline workload: all queries of a benchmark in one call
        _search("bulk_10m_u8", "uint8", "l2", 10_000_000, 128, 10_000, 10, batch=10_240),
        # embeddings of 768 dimensions: bulk retrieval of long lists
        _search("bulk_wide_f32", "float32", "cosine", 1_000_000, 768, 10_000, 100, batch=10_240),
        # the filtered workload: every query searches the vectors of its own label; 1 % of the vectors were replaced
        {"name": "labels_wide_f32", "path": "labels", "dtype": "float32", "metric": "cosine", "n": 1_000_000, "dim": 768,
         "queries": 10_000, "k": 100, "labels": 64},
        # sparse attention, a batch of 16 decoding rows over a long cache of 8 KV heads and 32 query heads
        _cache("keys_batch", "keys", 131_072, 2048, 16),
        # one decoding step of one sequence on such a cache: a key per head comes in, the query heads ask
        _cache("decode_step", "decode", 131_072, 2048, 1),
        # a batch of sequences of different lengths, some shorter than k
        {"name": "select_ragged", "path": "select", "kv_heads": 8, "heads": 32, "dim": 128, "keys": 40_000, "sequences": 12,
         "k": 2048},
        # a prompt's keys as they come out of the model: cached, grouped by head and asked by its last rows
        _cache("prefill_keys", "prefill", 32_768, 1024, 4),
        # an index for one use: a set that is searched for its own neighbours once (deduplication, graph building)
        {"name": "one_call_f16", "path": "one_call", "dtype": "float16", "metric": "l2", "n": 200_000, "dim": 96,
         "queries": 5000, "k": 10},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, uniform in its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    path = rng.choice(["search", "search", "search", "labels", "keys", "decode", "prefill", "select", "one_call"])
    if path in ("keys", "decode", "prefill"):
        kv = rng.choice([1, 2, 4, 8])
        keys = _log(rng, 2500, 131_072)
        return {"path": path, "kv_heads": kv, "heads": kv * rng.choice([1, 2, 4, 8]), "dim": rng.choice([64, 80, 96, 128]),
                "keys": keys, "rows": 1 if path == "decode" else _log(rng, 1, 16), "k": min(_log(rng, 32, 2048), keys // 2)}
    if path == "select":
        kv = rng.choice([1, 2, 4, 8])
        return {"path": path, "kv_heads": kv, "heads": kv * rng.choice([1, 2, 4]), "dim": rng.choice([64, 128]),
                "keys": _log(rng, 2000, 40_000), "sequences": _log(rng, 1, 16), "k": _log(rng, 64, 2048)}
    dtype = rng.choice(["float32", "float16", "int8", "uint8"])
    metric = rng.choice(["l2", "ip"] if dtype in ("int8", "uint8") else ["l2", "ip", "cosine"])
    dim = rng.choice([_log(rng, 20, 1024), 64, 96, 128, 256, 768])
    k = _log(rng, 1, 200)
    if path == "labels":
        n, queries = _log(rng, 50_000, 1_000_000), _log(rng, 16, 10_000)
        return {"path": path, "dtype": dtype, "metric": metric, "n": n, "dim": dim, "queries": queries, "k": k,
                "labels": _log(rng, 4, 256)}
    n = _log(rng, 2000, 300_000 if path == "one_call" else 2_000_000)
    # small sets and long lists are scored whole: fewer queries there, so that no drawn case outweighs the listed ones
    limit = 1e11 if n < 256 * k else 4e12
    queries = _log(rng, 1, 10_000)
    if path == "one_call":
        queries = min(queries, max(1, int(limit / (2 * n * dim))))
        return {"path": path, "dtype": dtype, "metric": metric, "n": n, "dim": dim, "queries": queries, "k": k}
    kept = rng.choice(["none", "none", "bitset", "bitmap"])
    if kept == "bitmap":
        n, queries, limit = min(n, 200_000), min(queries, 400), 2e10
    queries = min(queries, max(1, int(limit / (2 * n * dim))))
    return {"path": path, "dtype": dtype, "metric": metric, "n": n, "dim": dim, "queries": queries, "k": k, "filter": kept,
            "batch": rng.choice([2048, 10_240])}


# ------------------------------------------------------------------------------------------------------------ inputs
def _vectors(dtype, metric, n, dim, seed):
    """Rows of the package's own synthetic sets: a mixture of bytes, unit vectors in clusters (cosine), Gaussian
    rows for the other float searches."""
    if dtype in ("int8", "uint8"):
        x = synthetic.mixture_u8(n, dim, seed=seed)
        return x if dtype == "uint8" else (x.to(torch.int16) - 128).to(torch.int8)
    if metric == "cosine":
        return synthetic.clustered_unit_f32(n, dim, seed=seed).to(_DTYPES[dtype])
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((n, dim), generator=g, device="cuda").to(_DTYPES[dtype])


def _ints(hi, n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(0, hi, (n,), generator=g, dtype=torch.int32, device="cuda")


def _tokens(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16)


def _lengths(case):
    """Sequence lengths of a "select" case: from a thirtieth of `keys` to all of it, no two alike."""
    rng = random.Random(case["keys"] * 31 + case["sequences"])
    return [max(1, _log(rng, case["keys"] // 30, case["keys"])) for _ in range(case["sequences"] - 1)] + [case["keys"]]


def prepare(case, seed):
    path = case["path"]
    state = {"case": case}
    if path in ("keys", "decode", "prefill"):
        n, spare = case["keys"], _STEPS if path == "decode" else 0
        keys = synthetic.keys_with_outliers(case["kv_heads"], n + spare, case["dim"], seed=2 * seed)
        state["q"] = _tokens((case["heads"], case["rows"], case["dim"]), 2 * seed + 1)
        if path == "prefill":
            return dict(state, keys=keys)
        # room for the keys of a long answer, as a server reserves it
        room = n + (1 << 14) if spare else n
        state["cache"] = certex.KeyCache(case["kv_heads"], case["dim"], k=case["k"], capacity=room).append(keys[:, :n].contiguous())
        if path == "decode":
            state.update(new=[keys[:, i : i + 1].contiguous() for i in range(n, n + _STEPS)], step=0)
        return state
    if path == "select":
        select = flashinfer.ExactTopK(case["kv_heads"], case["dim"], k_max=case["k"], capacity=sum(_lengths(case)))
        for slot, n in enumerate(_lengths(case)):
            select.append(slot, _tokens((n, case["kv_heads"], case["dim"]), 1000 * seed + slot))
        state.update(select=select, q=_tokens((case["sequences"], case["heads"], case["dim"]), 1000 * seed + 999))
        return state
    n, dim, metric = case["n"], case["dim"], case["metric"]
    x = _vectors(case["dtype"], metric, n, dim, 2 * seed)
    state["q"] = _vectors(case["dtype"], metric, case["queries"], dim, 2 * seed + 1)
    if path == "one_call":
        return dict(state, x=x)
    changed = n // 100 if path == "labels" else 0
    index = certex.Index(dim, metric=metric, capacity=n + changed)
    if path == "labels":
        index.add(x, labels=_ints(case["labels"], n, seed))
        gone = torch.arange(seed % 97, n, 100, device="cuda")[:changed]
        index.remove(gone)
        index.add(_vectors(case["dtype"], metric, changed, dim, 2 * seed + 7), labels=_ints(case["labels"], changed, seed + 1))
        state["labels"] = _ints(case["labels"], case["queries"], seed + 2)
    else:
        index.add(x)
        g = torch.Generator(device="cuda").manual_seed(seed + 3)
        shape = {"none": None, "bitset": (n,), "bitmap": (case["queries"], n)}[case["filter"]]
        state["mask"] = None if shape is None else torch.rand(shape, generator=g, device="cuda") < 0.5
    return dict(state, index=index)


# -------------------------------------------------------------------------------------------------------------- calls
def run(state):
    case = state["case"]
    path, k = case["path"], case["k"]
    if path == "search":
        return state["index"].search(state["q"], k=k, batch=case["batch"], filter=state["mask"], return_scores=True)
    if path == "labels":
        return state["index"].search(state["q"], k=k, batch=10_240, labels=state["labels"], return_scores=True)
    if path == "keys":
        return state["cache"].topk(state["q"], k)
    if path == "decode":
        state["cache"].append(state["new"][state["step"] % _STEPS])
        state["step"] += 1
        return state["cache"].topk(state["q"], k)
    if path == "prefill":
        return certex.topk(state["q"], state["keys"], k)
    if path == "select":
        return state["select"].select(state["q"], k)
    return certex.search(state["x"], state["q"], k=k, metric=case["metric"])


# --------------------------------------------------------------------------------------------------------------- work
def work(case):
    """Bytes: the stored vectors once (floats as two bytes a coordinate, which is what a first look at them takes), for
    every neighbour that is returned its vector as it is stored, the queries, masks and results. Operations: a product and
    a sum per coordinate of every pair of a query and a vector it may return."""
    path, k = case["path"], case["k"]
    if path in ("keys", "decode", "prefill", "select"):
        # every query head looks at the keys of one KV head of its sequence
        lengths = _lengths(case) if path == "select" else [case["keys"]]
        rows = case.get("rows", 1)
        row = 2 * case["dim"]
        pairs = sum(case["heads"] * rows * n for n in lengths)
        found = sum(case["heads"] * rows * min(k, n) for n in lengths)
        return {"bytes": sum(lengths) * case["kv_heads"] * row + found * (row + (4 if path == "select" else 12)),
                "flops": 2.0 * pairs * case["dim"]}
    size, nq, n = _BYTES[case["dtype"]], case["queries"], case["n"]
    first = min(size, 2)
    pairs = float(nq) * n / (case["labels"] if path == "labels" else 1)
    bits = {"bitset": n, "bitmap": nq * n}.get(case.get("filter"), 0)  # a mask arrives as one byte per entry
    read = n * case["dim"] * (size if path == "one_call" else first)
    return {"bytes": read + bits + nq * case["dim"] * size + nq * k * (case["dim"] * size + 20), "flops": 2.0 * pairs * case["dim"]}


def tolerance(case):
    """Every answer is the exact one: the neighbours by their fp64 score (sums in coordinate order, every operation rounded
    on its own), equal scores by the smaller id, and the distances that follow from those scores."""
    return "exact"
