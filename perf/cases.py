"""Performance cases: what a user of this library has it do, through its public entry points.

A case is a dict of plain values.  `kind` names the call:

  multiselect  many k's of a device vector, in one call (ggks.multiselect)
  select       one k of a device vector (bucketSelectWrapper)
  topk         the K largest of a device vector (ggks.topk)
  host         many k's of a vector in pinned host memory (multiselect_host): the whole call,
               the copy over the link included
  batch        a batched multiselect / top-k over device vectors of uneven lengths
               (PreparedBatch, whose argument arrays a program keeps)
  serve        a burst of mixed requests to a running server: submit all, wait for all

Every output is an order statistic, so a value is right only if it is the value that sorting
and indexing gives (`exact`).
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("ggks-multiselect_gb300"))
import ggks  # noqa: E402

_NP = {"f32": np.float32, "f64": np.float64, "u32": np.uint32}
_TORCH = {"f32": torch.float32, "f64": torch.float64, "u32": torch.int32}  # u32: the bits
_SIZE = {"f32": 4, "f64": 8, "u32": 4}
_FLOAT_DISTS = ("uniform", "normal", "half_normal", "cauchy", "small_ints")


def listed():
    return [
        # a statistics call inside a loop over small blocks: deciles and extremes of a few
        # thousand values, where the call's latency is everything
        {"name": "tiny_f32", "kind": "multiselect", "dtype": "f32", "dist": "normal", "n": 5003,
         "num_k": 11, "skip": 0},
        # the plain configuration: every percentile of 2^20 uniform floats
        {"name": "percentiles_f32", "kind": "multiselect", "dtype": "f32", "dist": "uniform",
         "n": 1 << 20, "num_k": 101, "skip": 0},
        # an ordinary column of a data set: ragged length, heavy tails, a slice that starts off
        # a 16-byte boundary
        {"name": "column_f32", "kind": "multiselect", "dtype": "f32", "dist": "cauchy",
         "n": 10_000_019, "num_k": 257, "skip": 1},
        # the large configuration: 1001 order statistics of 2^28 normal floats
        {"name": "large_f32", "kind": "multiselect", "dtype": "f32", "dist": "normal",
         "n": 1 << 28, "num_k": 1001, "skip": 0},
        # the large configuration in double precision (scientific data)
        {"name": "large_f64", "kind": "multiselect", "dtype": "f64", "dist": "uniform",
         "n": 1 << 27, "num_k": 1001, "skip": 0},
        # integer data with many copies of each value (counts, pixel values, quantised codes)
        {"name": "duplicates_u32", "kind": "multiselect", "dtype": "u32", "dist": "u16",
         "n": (1 << 26) + 3, "num_k": 1001, "skip": 0},
        # a median (thresholds, robust statistics)
        {"name": "median_f32", "kind": "select", "dtype": "f32", "dist": "normal",
         "n": 50_000_017, "at": 0.5, "skip": 0},
        # the top-k configuration, a short list (search results, gradient sparsification)
        {"name": "topk_f32", "kind": "topk", "dtype": "f32", "dist": "uniform", "n": 1 << 26,
         "num_k": 1024, "skip": 0},
        # the top-k configuration, a long list from duplicate-heavy integers
        {"name": "topk_long_u32", "kind": "topk", "dtype": "u32", "dist": "u16", "n": 1 << 26,
         "num_k": 65536, "skip": 0},
        # the batched configuration: thousands of independent vectors of uneven lengths
        {"name": "batch_f32", "kind": "batch", "dtype": "f32", "count": 4096, "lo": 1 << 10,
         "hi": 1 << 22, "max_k": 64, "top": False, "packed": False},
        # a vector that lives in pinned host memory (an ingest path, a data loader)
        {"name": "host_f32", "kind": "host", "dtype": "f32", "dist": "normal", "n": 1 << 26,
         "num_k": 101},
        # the serving configuration's request mix, as one burst to a running server
        {"name": "serve_mixed", "kind": "serve", "count": 96, "lo": 1 << 12, "hi": 1 << 26},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _draw_values(rng):
    """An element type and a distribution that the types meet in use."""
    dtype = rng.choice(("f32", "f32", "f32", "u32", "f64"))
    if dtype == "u32":
        return dtype, rng.choice(("uniform", "u16"))
    if dtype == "f64":
        return dtype, rng.choice(("uniform", "normal"))
    return dtype, rng.choice(_FLOAT_DISTS + ("ascending",))


def draw(rng):
    kind = rng.choice(("multiselect",) * 5 + ("topk",) * 3 + ("select", "host", "batch", "serve"))
    if kind == "batch":
        count = _log_int(rng, 16, 4096)
        lo = _log_int(rng, 1 << 10, 1 << 14)
        hi = _log_int(rng, 1 << 16, 1 << 22)
        return {"kind": kind, "dtype": rng.choice(("f32", "f32", "u32", "f64")), "count": count,
                "lo": lo, "hi": hi if count <= 1024 else min(hi, 1 << 20),
                "max_k": _log_int(rng, 1, 64), "top": rng.random() < 0.3,
                "packed": rng.random() < 0.5}
    if kind == "serve":
        return {"kind": kind, "count": _log_int(rng, 8, 96), "lo": 1 << 12,
                "hi": _log_int(rng, 1 << 18, 1 << 26)}
    dtype, dist = _draw_values(rng)
    if kind == "host":
        n = _log_int(rng, 1 << 16, 1 << 26)
        return {"kind": kind, "dtype": dtype, "dist": dist, "n": n,
                "num_k": _log_int(rng, 1, 1001)}
    skip = rng.choice((0, 0, 1, 3))
    if kind == "select":
        return {"kind": kind, "dtype": dtype, "dist": dist, "n": _log_int(rng, 1 << 12, 1 << 27),
                "at": rng.uniform(0.0, 1.0), "skip": skip}
    if kind == "topk":
        n = _log_int(rng, 1 << 14, 1 << 26)
        return {"kind": kind, "dtype": dtype, "dist": dist, "n": n,
                "num_k": min(n // 16, _log_int(rng, 8, 65536)), "skip": skip}
    n = _log_int(rng, 1 << 12, 1 << (27 if dtype == "f64" else 28))
    return {"kind": kind, "dtype": dtype, "dist": dist, "n": n,
            "num_k": min(n // 4, _log_int(rng, 3, 1001)), "skip": skip}


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------


def _fill(t, dtype, dist, gen):
    """Fills a device tensor with values of a distribution, in place.  The ranges of the
    few-valued ones depend on the seed a little, so that their extremes and medians do."""
    few = gen.initial_seed() % 61
    if dtype == "u32":
        if dist == "u16":
            t.random_(0, (1 << 16) - few, generator=gen)
        else:
            t.random_(-(1 << 31), 1 << 31, generator=gen)
    elif dist in ("uniform", "ascending"):
        if dtype == "f64":
            t.uniform_(-1e6, 1e6, generator=gen)
        else:
            t.uniform_(0.0, 1.0, generator=gen)
        if dist == "ascending":
            t.copy_(torch.sort(t).values)
    elif dist in ("normal", "half_normal"):
        t.normal_(0.0, 1.0, generator=gen)
        if dist == "half_normal":
            t.abs_()
    elif dist == "cauchy":
        t.cauchy_(generator=gen)
    elif dist == "small_ints":
        t.random_(0, 256 - few, generator=gen)
    else:
        raise ValueError(dist)


def _vector(case, seed):
    """The case's device vector: a slice that starts `skip` elements into its buffer."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    buf = torch.empty(case["n"] + case.get("skip", 0), dtype=_TORCH[case["dtype"]], device="cuda")
    v = buf[case.get("skip", 0):]
    _fill(v, case["dtype"], case["dist"], gen)
    return v


def _ks(rng, n, count):
    """`count` k's (k-th largest, 1-based) uniform over the vector."""
    return rng.integers(1, n + 1, size=count).astype(np.uint32)


def _lengths(count, lo, hi):
    """Lengths spread evenly over the logarithm of [lo, hi]; the same total for every seed."""
    return [int(lo * (hi / lo) ** ((i + 0.5) / count)) for i in range(count)]


def _batch_inputs(case, seed):
    """The batch's vectors (in runs of one distribution each) and its k lists or K's."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = np.array(_lengths(case["count"], case["lo"], case["hi"]), dtype=np.int64)
    rng.shuffle(n)
    slot = n if case["packed"] else (n + 63) // 64 * 64
    start = np.concatenate([[0], np.cumsum(slot)])
    buf = torch.empty(int(start[-1]), dtype=_TORCH[case["dtype"]], device="cuda")
    dists = {"f32": ("uniform", "normal", "cauchy", "small_ints"), "u32": ("uniform", "u16"),
             "f64": ("uniform", "normal")}[case["dtype"]]
    cut = [case["count"] * i // len(dists) for i in range(len(dists) + 1)]
    for i, dist in enumerate(dists):
        _fill(buf[int(start[cut[i]]):int(start[cut[i + 1]])], case["dtype"], dist, gen)
    vecs = [buf[int(s):int(s + m)] for s, m in zip(start, n)]
    num = [1 + i % case["max_k"] for i in range(case["count"])]
    order = rng.permutation(case["count"])  # the caller's order mixes lengths and distributions
    return [vecs[i] for i in order], [_ks(rng, len(vecs[i]), num[i]) for i in order]


def _serve_inputs(case, seed):
    """The burst's requests: (dtype, vector, k list or None, K)."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    reqs = []
    for i, n in enumerate(_lengths(case["count"], case["lo"], case["hi"])):
        dtype = ("f32", "u32", "f32", "f64", "f32", "u32", "f32", "f32", "u32", "f32")[i % 10]
        dists = {"f32": _FLOAT_DISTS, "u32": ("uniform", "u16"), "f64": ("uniform", "normal")}[dtype]
        t = torch.empty(n, dtype=_TORCH[dtype], device="cuda")
        _fill(t, dtype, dists[i // 10 % len(dists)], gen)
        if i % 3 == 2:
            reqs.append((dtype, t, None, min(n, 16 << (i % 9))))
        else:
            count = 8 << (i % 8)
            reqs.append((dtype, t, _ks(rng, n, count), count))
    return [reqs[i] for i in rng.permutation(len(reqs))]


def prepare(case, seed):
    state = {"case": case}
    rng = np.random.default_rng(seed + 1)
    kind = case["kind"]
    if kind in ("multiselect", "topk", "select"):
        state["vec"] = _vector(case, seed)
        if kind == "multiselect":
            state["k"] = _ks(rng, case["n"], case["num_k"])
    elif kind == "host":
        v = _vector(case, seed)
        pinned = torch.empty(v.shape, dtype=v.dtype, pin_memory=True)
        pinned.copy_(v)
        state["pinned"] = pinned
        state["vec"] = pinned.numpy().view(_NP[case["dtype"]])
        state["k"] = _ks(rng, case["n"], case["num_k"])
    elif kind == "batch":
        vecs, ks = _batch_inputs(case, seed)
        lists = {"Ks": [len(k) for k in ks]} if case["top"] else {"k_lists": ks}
        state["vecs"] = vecs
        state["batch"] = ggks.PreparedBatch([v.data_ptr() for v in vecs], [len(v) for v in vecs],
                                            _NP[case["dtype"]], **lists)
    else:
        reqs = _serve_inputs(case, seed)
        state["reqs"] = reqs
        state["server"] = ggks.Server(device=0, hbm_cap_bytes=64 << 30)
        state["out"] = {d: np.empty(sum(r[3] for r in reqs if r[0] == d), dtype=_NP[d])
                        for d in sorted({r[0] for r in reqs})}
        at = dict.fromkeys(state["out"], 0)
        state["slices"] = []
        for d, _, _, count in reqs:
            state["slices"].append(state["out"][d][at[d]:at[d] + count])
            at[d] += count
    torch.cuda.synchronize()  # the library's calls run on its own stream
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "multiselect":
        return ggks.multiselect(state["vec"], state["k"])
    if kind == "topk":
        return ggks.topk(state["vec"], case["num_k"])
    if kind == "select":
        return ggks.bucketSelectWrapper(state["vec"], case["n"], _select_k(case))
    if kind == "host":
        return ggks.multiselect_host(state["vec"], state["k"])
    if kind == "batch":
        return state["batch"]()
    server = state["server"]
    tickets = []
    for (dtype, t, k, count), out in zip(state["reqs"], state["slices"]):
        tickets.append(server.submit(t.data_ptr(), t.numel(), _NP[dtype], k=k,
                                     K=count if k is None else None, out=out))
    for ticket in tickets:
        server.wait(ticket)
    return state["out"]


def _select_k(case):
    return 1 + int(case["at"] * (case["n"] - 1))


def work(case):
    """Every element of every vector read once, every k read and every value written once."""
    kind = case["kind"]
    if kind == "serve":
        total = 0
        for i, n in enumerate(_lengths(case["count"], case["lo"], case["hi"])):
            size = 8 if i % 10 == 3 else 4
            count = min(n, 16 << (i % 9)) if i % 3 == 2 else 8 << (i % 8)
            total += n * size + count * (size + (0 if i % 3 == 2 else 4))
        return {"bytes": total, "flops": 0}
    size = _SIZE[case["dtype"]]
    if kind == "batch":
        outs = sum(1 + i % case["max_k"] for i in range(case["count"]))
        elements = sum(_lengths(case["count"], case["lo"], case["hi"]))
        return {"bytes": elements * size + outs * (size + (0 if case["top"] else 4)), "flops": 0}
    outs = 1 if kind == "select" else case["num_k"]
    ks = 0 if kind in ("select", "topk") else 4 * outs
    return {"bytes": case["n"] * size + outs * size + ks, "flops": 0}


# ------------------------------------------------------------------------------------------------
# what sorting and indexing gives
# ------------------------------------------------------------------------------------------------


def _pick(v, dtype, k=None, K=None):
    """The k-th largest values, or the K largest in descending order, of a device vector."""
    if dtype == "u32":
        v = v.to(torch.int64) & 0xFFFFFFFF
    s = torch.sort(v).values
    if K is not None:
        got = s[len(s) - K:].flip(0)
    else:
        got = s[torch.from_numpy(len(s) - k.astype(np.int64)).to(s.device)]
    return got if dtype == "u32" else got.to(torch.float64)


def exact(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed + 1)
    if kind in ("multiselect", "host"):
        v = _vector(case, seed)
        return _pick(v, case["dtype"], k=_ks(rng, case["n"], case["num_k"]))
    if kind == "select":
        got = _pick(_vector(case, seed), case["dtype"], k=np.array([_select_k(case)]))
        return got[0]
    if kind == "topk":
        return _pick(_vector(case, seed), case["dtype"], K=case["num_k"])
    if kind == "batch":
        vecs, ks = _batch_inputs(case, seed)
        return torch.cat([_pick(v, case["dtype"], **({"K": len(k)} if case["top"] else {"k": k}))
                          for v, k in zip(vecs, ks)])
    found = {}
    for dtype, t, k, count in _serve_inputs(case, seed):
        found.setdefault(dtype, []).append(_pick(t, dtype, k=k, K=count if k is None else None))
    return {d: torch.cat(x) for d, x in sorted(found.items())}
