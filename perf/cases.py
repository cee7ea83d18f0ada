"""The work a user of this package has it do, as timed cases through the public API.

A case names the operation (`op`), the data it meets (`data`), the table's shape in words and
the call's own sizes.  Values are made on the GPU from the seed alone:

  graph      float32 N(0, 0.3^2), low 15 mantissa bits cleared, 30% zeros (graph features)
  plain      float32 N(0, 0.5^2), 5% of the rows redrawn from N(0, 100^2)
  features   graph, with a scale 2^-k of each column's own and a quarter of them non-negative
  clusters   float32 mixture of 16 Gaussians with per-cluster scale 10^U(-3, 1) (embeddings)
  half       float16 N(0, 0.02^2) kept to 5 mantissa bits, 5% of the rows 200 times as large
  masked     words with a random set of invariant bits (`frac` of them); one row in ten has
             one word in five off the pattern
"""
import math

import numpy as np
import torch

import invariantbitpacking_b200 as ibp
from invariantbitpacking_b200.batch import BatchFetcher, SetRegistry

_INT = {1: torch.int8, 2: torch.int16, 4: torch.int32, 8: torch.int64}

# Stored bytes of a row over its raw bytes under the data's own mask, used for `work` alone.
_STORED = {"graph": 0.52, "features": 0.45, "plain": 0.97, "clusters": 0.95, "half": 0.7}


def listed():
    return [
        # a mini-batch of graph node features gathered from a table in host memory
        {"name": "host_fetch", "op": "fetch", "where": "host", "data": "graph", "wb": 8,
         "rows": 600_000, "words": 64, "count": 100_000, "zipf": 1.1},
        # a small request against a small host table, where latency counts
        {"name": "host_fetch_small", "op": "fetch", "where": "host", "data": "plain", "wb": 8,
         "rows": 16_384, "words": 128, "count": 2048, "zipf": 0.0},
        # a large mini-batch of graph features from a table kept compressed in HBM
        {"name": "device_fetch", "op": "fetch", "where": "device", "data": "graph", "wb": 8,
         "rows": 2_400_000, "words": 64, "count": 400_000, "zipf": 1.1},
        # one embedding lookup from one table in HBM: a few launches long
        {"name": "device_fetch_small", "op": "fetch", "where": "device", "data": "clusters",
         "wb": 8, "rows": 200_000, "words": 32, "count": 2048, "zipf": 1.05},
        # decompression of a whole set in HBM, 1 KiB rows of 32-bit words
        {"name": "device_set", "op": "set", "where": "device", "data": "masked", "wb": 4,
         "rows": 100_000, "words": 256, "frac": 0.5},
        # decompression of a whole set of 4 KiB rows (weights or cache pages kept packed)
        {"name": "device_set_long", "op": "set", "where": "device", "data": "masked", "wb": 8,
         "rows": 40_000, "words": 512, "frac": 0.75},
        # one lookup in each of 26 host tables, batched into one captured launch
        {"name": "tables_batch", "op": "batch", "data": "clusters", "wb": 8, "tables": 26,
         "rows": 200_000, "words": 32, "count": 2048, "zipf": 1.05},
        # the mask of a feature table, thresholds swept
        {"name": "preprocess", "op": "preprocess", "data": "features", "wb": 8, "rows": 600_000,
         "words": 64, "threshold": -1.0},
        # compressed size of every row of a table of 16-bit values, with the running total
        {"name": "sizes_half", "op": "sizes", "data": "half", "wb": 2, "rows": 1_000_000,
         "words": 128},
        # a block of new feature rows compressed where it lies
        {"name": "compress_inplace", "op": "inplace", "data": "graph", "wb": 8,
         "rows": 600_000, "words": 64},
        # rows of an odd length packed back to back, and a batch read back from them
        {"name": "condensed", "op": "condensed", "data": "masked", "wb": 4, "rows": 200_000,
         "words": 99, "frac": 0.6, "count": 50_000, "zipf": 0.0},
        # per-cluster masks of one embedding table
        {"name": "kmeans", "op": "kmeans", "data": "clusters", "wb": 8, "rows": 200_000,
         "words": 32, "centroids": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shape(rng, wb, max_bytes, min_words=8, max_words=1024, min_rows=500):
    """Words per row (odd ones and whole 16-byte ones alike) and rows within max_bytes."""
    words = _log(rng, min_words, max_words)
    if rng.random() < 0.5:
        words = max(words // 32, 1) * 32
    return words, _log(rng, min_rows, max(min_rows, min(max_bytes // (words * wb), 2_400_000)))


def draw(rng):
    op = rng.choice(["fetch", "fetch", "set", "set", "batch", "preprocess", "sizes", "inplace",
                     "condensed", "kmeans"])
    if op in ("preprocess", "sizes"):
        wb = rng.choice([1, 2, 4, 8])
        words, rows = _shape(rng, wb, 256 << 20)
        data = rng.choice(["masked", "features" if op == "preprocess" else "plain"])
        if wb < 4:
            data = rng.choice(["masked", "half"]) if op == "sizes" and wb == 2 else "masked"
        case = {"op": op, "data": data, "wb": wb, "rows": rows, "words": words}
        if data == "masked":
            case["frac"] = round(rng.uniform(0.3, 0.9), 3)
        if op == "preprocess":
            case["threshold"] = rng.choice([-1.0, 0.7, 0.9])
        return case
    wb = rng.choice([4, 8, 8])
    if op == "kmeans":
        words, rows = _shape(rng, wb, 48 << 20, 8, 64)
        return {"op": op, "data": "clusters", "wb": wb, "rows": rows, "words": words,
                "centroids": rng.randint(2, 16)}
    if op == "batch":
        words = rng.choice([16, 32, 33, 64, 100])
        return {"op": op, "data": "clusters", "wb": wb, "tables": rng.randint(2, 26),
                "rows": _log(rng, 10_000, 100_000), "words": words,
                "count": _log(rng, 256, 2048), "zipf": rng.choice([0.0, 1.05])}
    data = rng.choice(["graph", "plain", "masked"])
    frac = {"frac": round(rng.uniform(0.3, 0.97), 3)} if data == "masked" else {}
    if op == "set":
        words, rows = _shape(rng, wb, 160 << 20)
        return {"op": op, "where": "device", "data": data, "wb": wb, "rows": rows,
                "words": words, **frac}
    if op == "inplace":
        words, rows = _shape(rng, wb, 256 << 20)
        return {"op": op, "data": data, "wb": wb, "rows": rows, "words": words, **frac}
    words, rows = _shape(rng, wb, 300 << 20, min_rows=2000)
    count = _log(rng, 256, max(256, min(400_000, (100 << 20) // (words * wb))))
    zipf = rng.choice([0.0, 1.05, 1.1])
    if op == "condensed":
        data, frac = "masked", {"frac": round(rng.uniform(0.3, 0.97), 3)}
        rows = min(rows, max(2000, (80 << 20) // (words * wb)))
        return {"op": op, "data": data, "wb": wb, "rows": rows, "words": words,
                "count": min(count, 100_000), "zipf": zipf, **frac}
    return {"op": op, "where": rng.choice(["host", "device", "device"]), "data": data, "wb": wb,
            "rows": rows, "words": words, "count": count, "zipf": zipf, **frac}


# ---------------------------------------------------------------------------- inputs
def _normal(g, n, cols, std, dtype=torch.float32):
    x = torch.randn((n, cols), generator=g, device="cuda", dtype=torch.float32)
    return (x * std).to(dtype)


def _words(x, wb):
    return x.contiguous().view(torch.uint8).view(_INT[wb])


def _rows(case, g, rows=None):
    """The case's raw rows, [rows, words] of `wb`-byte integers on the GPU."""
    n, v, wb = rows or case["rows"], case["words"], case["wb"]
    data = case["data"]
    if data == "half":
        x = _normal(g, n, (v * wb + 1) // 2, 0.02, torch.float16).view(torch.int16) & -32
        x = x.view(torch.float16)
        x[torch.rand(n, generator=g, device="cuda") < 0.05] *= 200.0
        return x.view(torch.uint8)[:, :v * wb].contiguous().view(_INT[wb])
    if data == "masked":
        return _masked(case, g, n)
    cols = v * wb // 4
    if data in ("graph", "features"):
        x = _normal(g, n, cols, 0.3)
        if data == "features":
            x *= 2.0 ** -torch.randint(0, 8, (cols,), generator=g, device="cuda")
            plus = torch.rand(cols, generator=g, device="cuda") < 0.25
            x = torch.where(plus, x.abs(), x)
        x = x.view(torch.int32) & -32768
        x[torch.rand((n, cols), generator=g, device="cuda") < 0.3] = 0
    elif data == "plain":
        x = _normal(g, n, cols, 0.5)
        far = torch.rand(n, generator=g, device="cuda") < 0.05
        x[far] *= 200.0
    else:
        cent = torch.randn((16, cols), generator=g, device="cuda")
        scale = 10.0 ** (torch.rand(16, generator=g, device="cuda") * 4 - 3)
        lab = torch.randint(0, 16, (n,), generator=g, device="cuda")
        x = _normal(g, n, cols, 1.0) * scale[lab, None] + cent[lab]
    return _words(x, wb)


def _masked(case, g, n):
    """Every word keeps the same number of bits and a tenth of the rows has the same number of
    words off the pattern, so that a set's compressed bytes depend on its shape alone."""
    v, wb = case["words"], case["wb"]
    bits = 8 * wb
    order = torch.rand((v, bits), generator=g, device="cuda").argsort(1)
    m = torch.zeros(v, dtype=torch.int64, device="cuda")
    off = torch.zeros(v, dtype=torch.int64, device="cuda")
    for b in range(bits):
        bit = (1 << b) if b < 63 else -(1 << 63)
        m |= (order[:, b] < round(case["frac"] * bits)).to(torch.int64) * bit
        off |= (order[:, b] == 0).to(torch.int64) * bit  # the invariant bit that goes wrong
    lo, hi = torch.iinfo(torch.int64).min, torch.iinfo(torch.int64).max
    base = torch.randint(lo, hi, (v,), generator=g, device="cuda") & m
    x = (torch.randint(lo, hi, (n, v), generator=g, device="cuda") & ~m) | base
    rows = torch.randperm(n, generator=g, device="cuda")[:n // 10]
    shift = torch.randint(0, v, (rows.numel(), 1), generator=g, device="cuda")
    stray = (torch.arange(v, device="cuda") + shift) % v < v // 5
    x[rows] ^= torch.where(stray, off, torch.zeros_like(off))
    return x.to(_INT[wb])  # the low bits of each word


def _index(case, g, rows=None):
    """`count` row ids, Zipf(s) over a random order of the rows (distinct where s is 0)."""
    n, k, s = rows or case["rows"], case["count"], case["zipf"]
    perm = torch.randperm(n, generator=g, device="cuda")
    if s == 0.0:
        return perm[torch.arange(k, device="cuda") % n].contiguous()
    cdf = torch.cumsum(torch.arange(1, n + 1, dtype=torch.float64, device="cuda") ** -s, 0)
    u = torch.rand(k, generator=g, device="cuda", dtype=torch.float64) * cdf[-1]
    return perm[torch.searchsorted(cdf, u).clamp_(max=n - 1)].contiguous()


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _pinned(x):
    out = torch.empty(x.shape, dtype=x.dtype, pin_memory=True)
    out.copy_(x)
    return out


def _packed(x):
    """What a program keeps of a set: its rows compressed in place, and how to read them."""
    mask, bitval = ibp.preprocess(x, 0.9)
    comp_len = ibp.get_single_compress_len(x, mask, bitval)
    bitmask = ibp.compress_inplace(x, mask, bitval)
    return {"comp": x, "mask": mask, "bitval": bitval, "bitmask": bitmask, "comp_len": comp_len}


def prepare(case, seed):
    g = _gen(seed)
    op = case["op"]
    if op in ("fetch", "set"):
        st = _packed(_rows(case, g))
        st["index"] = _index(case, g) if op == "fetch" else None
        if case["where"] == "host":
            st["comp"] = _pinned(st["comp"])
    elif op == "batch":
        sets, reqs = [], []
        for t, n in enumerate(_table_rows(case)):
            p = _packed(_rows(case, g, n))
            sets.append((_pinned(p["comp"]), p["mask"], p["bitval"], p["bitmask"],
                         p["comp_len"]))
            reqs.append((t, _index(case, g, n), 0, case["count"]))
        fetcher = BatchFetcher(SetRegistry(sets), max_requests=len(reqs))
        fetcher.capture()
        st = {"fetcher": fetcher, "requests": reqs}
    else:
        x = _rows(case, g)
        st = {"rows": x}
        if op in ("sizes", "inplace", "condensed"):
            st["mask"], st["bitval"] = ibp.preprocess(x, 0.9)
        if op == "sizes":
            st["total"] = torch.zeros(1, dtype=torch.int64, device="cuda")
        elif op == "inplace":
            st["block"] = torch.empty_like(x)
        elif op == "condensed":
            st["index"] = _index(case, g)
        elif op == "kmeans":
            st["seeds"] = _seed_rows(case, seed)
    st["case"] = dict(case)
    torch.cuda.synchronize()
    return st


def _table_rows(case):
    """Row counts of the batched tables: spread over a factor of ten up to `rows`."""
    k = case["tables"]
    return [max(int(case["rows"] * 10 ** (-t / max(k - 1, 1))), 1000) for t in range(k)]


def _seed_rows(case, seed):
    rng = np.random.default_rng(seed)
    k = min(case["centroids"], case["rows"])
    return rng.choice(case["rows"], k, replace=False).astype(np.int64)


# ---------------------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    op = case["op"]
    if op in ("fetch", "set"):
        return ibp.decompress_fetch(state["comp"], state["mask"], state["bitval"],
                                    state["bitmask"], "cuda", state["comp_len"], state["index"])
    if op == "batch":
        return state["fetcher"].fetch(state["requests"])
    if op == "preprocess":
        t = case["threshold"]
        return ibp.preprocess(state["rows"], None if t < 0 else t)
    if op == "sizes":
        state["total"].zero_()
        sizes = ibp.get_compress_size(state["rows"], state["mask"], state["bitval"], None,
                                      state["total"])
        return sizes, state["total"]
    if op == "inplace":
        # new rows arrive in the block that is then compressed where it lies
        state["block"].copy_(state["rows"])
        bitmask = ibp.compress_inplace(state["block"], state["mask"], state["bitval"])
        return state["block"], bitmask
    if op == "condensed":
        comp, offsets = ibp.compress_condensed(state["rows"], state["mask"], state["bitval"])
        out = ibp.decompress_fetch_condensed(comp, offsets, state["mask"], state["bitval"],
                                             case["words"], "cuda", state["index"])
        return comp, offsets, out
    return ibp.preprocess_kmeans(state["rows"], case["centroids"], 0.9,
                                 seed_rows=state["seeds"])


def exact(case, seed):
    """Fetched rows are the rows that were stored; the other outputs (masks, sizes, packed
    rows) are whole numbers defined by the format alone."""
    op = case["op"]
    g = _gen(seed)
    if op == "set":
        return _rows(case, g)
    if op == "fetch":
        x = _rows(case, g)
        return x[_index(case, g)]
    if op == "condensed":
        x = _rows(case, g)
        return None, None, x[_index(case, g)]
    if op == "batch":
        outs = []
        for n in _table_rows(case):
            x = _rows(case, g, n)
            outs.append(x[_index(case, g, n)])
        return outs
    return None


# ---------------------------------------------------------------------------- what a pass needs
def _distinct(n, k, s):
    """Expected distinct rows among k draws."""
    if s == 0.0:
        return min(n, k)
    p = np.arange(1, n + 1, dtype=np.float64) ** -s
    p /= p.sum()
    return float(-np.expm1(k * np.log1p(-np.minimum(p, 1 - 1e-12))).sum())


def work(case):
    """Bytes a pass cannot do without: each input read once, each output written once."""
    op = case["op"]
    raw = case["words"] * case["wb"]
    frac = _STORED.get(case["data"]) or min(1.0, 1.02 - case.get("frac", 0.0))
    stored = raw * frac
    n = case["rows"]
    if op == "set":
        nbytes = n * (stored + raw)
    elif op == "fetch":
        nbytes = _distinct(n, case["count"], case["zipf"]) * stored + case["count"] * (raw + 8)
    elif op == "batch":
        nbytes = sum(_distinct(m, case["count"], case["zipf"]) * stored +
                     case["count"] * (raw + 8) for m in _table_rows(case))
    elif op == "sizes":
        nbytes = n * (raw + 8)
    elif op == "inplace":
        nbytes = n * raw * 3 + n * raw  # the copy in, then the block read and rewritten
    elif op == "condensed":
        nbytes = n * (raw + stored + 8) + case["count"] * (stored + raw + 16)
    else:  # the masks need one pass over the rows, k-means reads them and writes a label each
        nbytes = n * raw + (4 * n if op == "kmeans" else 0)
    return {"bytes": int(nbytes), "flops": 0}
