"""The library's device-wide algorithms at the sizes, types and shapes they are used at.

A case is a dict of plain values.  ``op`` names the call; sizes, key and value
types and the inputs' distribution are the other entries.  ``listed()`` gives a
fixed set, ``draw(rng)`` one more from the same ranges:

* reduce, scan     2^10 to 2^28 elements of 4 bytes, to 2^27 of 8;
* merge            two sorted arrays of 2^10 to 2^27 elements in all, of any two
                   lengths, with and without a payload;
* sort             2^10 to 2^26 keys of 4 or 8 bytes, with and without a payload;
* reduce_by_key    2^10 to 2^27 pairs, geometric or Zipf run lengths;
* the batched forms of scan, sort and reduce_by_key, and the three together (a
  serving round), arrays of log-uniform lengths.

Every call goes through the package's public functions on the current stream
with the arguments a program would give; inputs are made on the GPU.
"""
import math
import random

import torch

import bulk_b200
from bulk_b200 import batch

DTYPES = {"i32": torch.int32, "u32": torch.uint32, "i64": torch.int64, "u64": torch.uint64,
          "f32": torch.float32, "f64": torch.float64}
SIZE = {"i32": 4, "u32": 4, "i64": 8, "u64": 8, "f32": 4, "f64": 8}
#: torch computes little on unsigned types: unsigned arrays are made and returned as signed ones of the same bytes
SIGNED = {"u32": torch.int32, "u64": torch.int64}


def listed():
    return [
        # the headline reduction, a plain sum over an array far larger than L2
        {"name": "reduce_f32_large", "op": "reduce", "key": "f32", "n": 1 << 28},
        # a prefix sum over a large array of ragged length, in the wide type
        {"name": "scan_f64_large_ragged", "op": "scan", "key": "f64", "n": (1 << 27) - 35},
        # a small prefix sum (offsets from counts): launches and the call itself
        {"name": "scan_i32_small", "op": "scan", "key": "i32", "n": 50_021},
        # the headline merge: two equal sorted float arrays with payloads
        {"name": "merge_by_key_f32_u32_large", "op": "merge", "key": "f32", "value": "u32", "n": 1 << 26, "m": 1 << 26},
        # a sorted table takes up a smaller sorted update, keys alone, ragged lengths
        {"name": "merge_i32_update", "op": "merge", "key": "i32", "value": None, "n": 3_000_017, "m": 700_001},
        # the headline sorts: 2^26 keys over the full range of their type, payload = original index
        {"name": "sort_u32_u32_large", "op": "sort", "key": "u32", "value": "u32", "n": 1 << 26},
        {"name": "sort_u64_u32_large", "op": "sort", "key": "u64", "value": "u32", "n": 1 << 26},
        # an ordinary sort by score, of ragged length
        {"name": "sort_f32_u32_medium", "op": "sort", "key": "f32", "value": "u32", "n": 1_000_003},
        # a small sort, as one serving request asks for
        {"name": "sort_i32_u32_small", "op": "sort", "key": "i32", "value": "u32", "n": 20_011},
        # the headline reduce_by_key: short geometric runs
        {"name": "reduce_by_key_i32_f32_large", "op": "reduce_by_key", "key": "i32", "value": "f32", "n": 1 << 27,
         "runs": "geometric"},
        # heavy-tailed runs, some longer than any tile, wide values, ragged length
        {"name": "reduce_by_key_i32_f64_zipf", "op": "reduce_by_key", "key": "i32", "value": "f64", "n": 5_000_011,
         "runs": "zipf"},
        # one round of the serving mix (40 % sorts, 30 % reduce_by_key, 30 % scans), all three batched calls
        {"name": "serving_round", "op": "round", "count": 30, "lo": 1 << 10, "hi": 1 << 22, "sizes": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["reduce", "scan", "merge", "merge", "sort", "sort", "sort", "reduce_by_key", "reduce_by_key",
                     "batch_scan", "batch_sort", "batch_reduce_by_key", "round"])
    if op in ("reduce", "scan"):
        key = rng.choice(["i32", "i64", "f32", "f64"])
        return {"op": op, "key": key, "n": _log(rng, 1 << 10, (1 << 30) // SIZE[key])}
    if op == "merge":
        key, value = rng.choice(["i32", "u32", "f32", "u64", "f64"]), rng.choice([None, "u32"])
        total, share = _log(rng, 1 << 10, 1 << (27 if SIZE[key] == 4 else 26)), rng.uniform(0.02, 0.98)
        return {"op": op, "key": key, "value": value, "n": int(total * share), "m": total - int(total * share)}
    if op == "sort":
        key, value = rng.choice(["i32", "u32", "f32", "i64", "u64", "f64"]), rng.choice([None, "u32", "u32", "u64"])
        return {"op": op, "key": key, "value": value, "n": _log(rng, 1 << 10, 1 << (26 if SIZE[key] == 4 else 25))}
    if op == "reduce_by_key":
        value = rng.choice(["f32", "f64"])
        return {"op": op, "key": rng.choice(["i32", "i32", "i64"]), "value": value, "n": _log(rng, 1 << 10, 1 << 26),
                "runs": rng.choice(["geometric", "zipf"])}
    return {"op": op, "count": rng.randint(6, 30), "lo": 1 << 10, "hi": _log(rng, 1 << 14, 1 << 22),
            "sizes": rng.randrange(1 << 20)}


# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _values(tag, n, g, unit=False):
    """Small integers, or uniform [-1, 1) ([0, 1) with ``unit``), as the sums are taken over."""
    if tag in ("i32", "i64"):
        return torch.randint(-100, 101, (n,), generator=g, device="cuda", dtype=DTYPES[tag])
    x = torch.rand(n, generator=g, device="cuda", dtype=DTYPES[tag])
    return x if unit else x * 2 - 1


def _keys(tag, n, g):
    """Sort keys: the whole range of an integer type, uniform [-1, 1) for a floating one (signed bytes for unsigned types)."""
    if tag in ("f32", "f64"):
        return _values(tag, n, g)
    k = torch.randint(-(1 << 31), 1 << 31, (n,), generator=g, device="cuda", dtype=torch.int64)
    if SIZE[tag] == 8:
        return (k << 32) ^ torch.randint(0, 1 << 32, (n,), generator=g, device="cuda", dtype=torch.int64)
    return k.to(torch.int32)


def _order(tag, keys):
    """64-bit values that torch sorts as the library sorts ``keys``."""
    if tag in ("f32", "f64"):
        return keys.double()
    if tag == "u32":
        return keys.long() & 0xFFFFFFFF
    if tag == "u64":
        return keys ^ -(1 << 63)
    return keys.long()


def _payload(tag, n):
    """The original index; a 4-byte one in signed bytes."""
    return torch.arange(n, device="cuda", dtype=torch.int32 if tag == "u32" else torch.int64)


def _typed(tag, t):
    return t.view(DTYPES[tag]) if tag in SIGNED else t


def _plain(tag, t):
    return t.view(SIGNED[tag]) if tag in SIGNED else t


def _sorted_keys(tag, n, g):
    """Sorted keys of which about 1 % are duplicated."""
    k = torch.rand(n, generator=g, device="cuda", dtype=DTYPES[tag]) if tag in ("f32", "f64") else _keys(tag, n, g)
    dup = torch.rand(n, generator=g, device="cuda") < 0.01
    k = torch.where(dup, k[torch.randint(0, max(n, 1), (n,), generator=g, device="cuda")], k)
    return k[torch.argsort(_order(tag, k))].contiguous()


def _runs(kind, tag, n, g, mean=16.0):
    """Run-index keys: geometric lengths of the given mean, or Zipf(1.2) lengths up to 2^20."""
    if kind == "geometric":
        new = torch.rand(n, generator=g, device="cuda") < 1.0 / mean
        return (torch.cumsum(new, 0) - new[:1].long()).to(DTYPES[tag])
    parts, have = [], 0
    weights = torch.arange(1, (1 << 20) + 1, device="cuda", dtype=torch.float64).pow_(-1.2).cumsum_(0)
    while have < n:
        u = torch.rand(max(1024, n // 64), generator=g, device="cuda", dtype=torch.float64) * weights[-1]
        lengths = torch.searchsorted(weights, u) + 1
        parts.append(lengths)
        have += int(lengths.sum())
    lengths = torch.cat(parts)
    ends = torch.cumsum(lengths, 0)
    new = torch.zeros(n, device="cuda", dtype=torch.int64)
    new[ends[ends < n]] = 1
    return torch.cumsum(new, 0).to(DTYPES[tag])


def _kinds(case):
    """The batched kinds of a case and how many arrays each has."""
    c = case["count"]
    if case["op"] == "round":
        return {"sort": c - 2 * (3 * c // 10), "reduce_by_key": 3 * c // 10, "scan": 3 * c // 10}
    return {case["op"][len("batch_"):]: c}


def _lengths(case):
    rng = random.Random(case["sizes"])
    return {k: [_log(rng, case["lo"], case["hi"]) for _ in range(c)] for k, c in _kinds(case).items()}


def _run_buffers(keys, vals):
    """Zeroed outputs of reduce_by_key, as long as its inputs: as many places as there are runs are written."""
    return torch.zeros_like(keys), torch.zeros_like(vals), torch.zeros(1, device="cuda", dtype=torch.int64)


def prepare(case, seed):
    g, op = _gen(seed), case["op"]
    if op in ("reduce", "scan"):
        return {"case": case, "x": _values(case["key"], case["n"], g)}
    if op == "merge":
        n, m = case["n"], case["m"]
        s = {"case": case, "a": _typed(case["key"], _sorted_keys(case["key"], n, g)),
             "b": _typed(case["key"], _sorted_keys(case["key"], m, g)), "av": None, "bv": None}
        if case["value"]:
            s["av"], s["bv"] = _payload(case["value"], n), _payload(case["value"], m) + n
        return s
    if op == "sort":
        s = {"case": case, "keys": _typed(case["key"], _keys(case["key"], case["n"], g)), "vals": None}
        if case["value"]:
            s["vals"] = _payload(case["value"], case["n"])
        return s
    if op == "reduce_by_key":
        keys = _runs(case["runs"], case["key"], case["n"], g)
        vals = _values(case["value"], case["n"], g, unit=True)
        return {"case": case, "keys": keys, "vals": vals, "outs": _run_buffers(keys, vals)}
    s = {"case": case}
    for kind, ns in _lengths(case).items():
        if kind == "scan":
            s[kind] = [_values("f32", n, g) for n in ns]
        elif kind == "sort":
            s[kind] = ([_typed("u32", _keys("u32", n, g)) for n in ns], [_payload("u32", n) for n in ns])
        else:
            keys = [_runs("geometric", "i32", n, g, 32.0) for n in ns]
            vals = [_values("f32", n, g, unit=True) for n in ns]
            s[kind] = (keys, vals)
            s["outs"] = [_run_buffers(k, v) for k, v in zip(keys, vals)]
    return s


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "reduce":
        return bulk_b200.reduce(state["x"])
    if op == "scan":
        return bulk_b200.inclusive_scan(state["x"])
    if op == "merge":
        out = bulk_b200.merge(state["a"], state["b"], state["av"], state["bv"])
        return (_plain(case["key"], out[0]), out[1]) if state["av"] is not None else _plain(case["key"], out)
    if op == "sort":  # the sort is in place: a program that keeps its table sorts a copy
        keys = state["keys"].clone()
        if state["vals"] is None:
            return _plain(case["key"], bulk_b200.stable_sort_by_key(keys))
        keys, vals = bulk_b200.stable_sort_by_key(keys, state["vals"].clone())
        return _plain(case["key"], keys), vals
    if op == "reduce_by_key":
        out_keys, out_vals, num_out = state["outs"]
        count = bulk_b200.reduce_by_key(state["keys"], state["vals"], out_keys, out_vals, num_out)[2]
        return out_keys, out_vals, count
    out = {}
    if "sort" in state:
        ks, vs = batch.stable_sort_by_key_copy_batch(*state["sort"])
        out["sort"] = [[_plain("u32", k) for k in ks], vs]
    if "scan" in state:
        out["scan"] = batch.inclusive_scan_batch(state["scan"])
    if "reduce_by_key" in state:
        batch.reduce_by_key_batch(*state["reduce_by_key"], sync=True, outs=state["outs"])
        out["reduce_by_key"] = [list(o[:2]) for o in state["outs"]]
    return out


# ---------------------------------------------------------------------------
def _split(x):
    """x as a whole multiple of 2^-30 and a rest below 2^-31: sums of the first part are exact in 64 bits."""
    hi = torch.round(x.double() * (1 << 30))
    return hi.long(), x.double() - hi / (1 << 30)


def _cumsum(x):
    if not x.is_floating_point():
        return torch.cumsum(x, 0, dtype=x.dtype)
    hi, lo = _split(x)
    return torch.cumsum(hi, 0).double() / (1 << 30) + torch.cumsum(lo, 0)


def _run_sums(keys, vals):
    last = torch.ones(keys.numel(), device="cuda", dtype=torch.bool)
    last[:-1] = keys[1:] != keys[:-1]
    ends = last.nonzero().reshape(-1)

    def each(v):
        c = torch.cumsum(v, 0)[ends]
        return torch.cat([c[:1], c[1:] - c[:-1]])

    def padded(v):
        return torch.cat([v, torch.zeros(keys.numel() - v.numel(), device="cuda", dtype=v.dtype)])

    hi, lo = _split(vals)
    return padded(keys[ends]), padded(each(hi).double() / (1 << 30) + each(lo)), ends.numel()


def exact(case, seed):
    s, op = prepare(case, seed), case["op"]
    if op == "reduce":
        x = s["x"]
        if not x.is_floating_point():
            return x.sum(dtype=torch.int64).to(x.dtype).reshape(1)
        hi, lo = _split(x)
        return (hi.sum().double() / (1 << 30) + lo.sum()).reshape(1)
    if op == "scan":
        return _cumsum(s["x"])
    if op == "merge":
        keys = torch.cat([_plain(case["key"], s["a"]), _plain(case["key"], s["b"])])
        order = torch.sort(_order(case["key"], keys), stable=True)[1]
        return (keys[order], torch.cat([s["av"], s["bv"]])[order]) if case["value"] else keys[order]
    if op == "sort":
        keys = _plain(case["key"], s["keys"])
        order = torch.sort(_order(case["key"], keys), stable=True)[1]
        return (keys[order], s["vals"][order]) if case["value"] else keys[order]
    if op == "reduce_by_key":
        return _run_sums(s["keys"], s["vals"])
    out = {}
    if "sort" in s:
        ks, vs = [_plain("u32", k) for k in s["sort"][0]], s["sort"][1]
        orders = [torch.sort(_order("u32", k), stable=True)[1] for k in ks]
        out["sort"] = [[k[o] for k, o in zip(ks, orders)], [v[o] for v, o in zip(vs, orders)]]
    if "scan" in s:
        out["scan"] = [_cumsum(x) for x in s["scan"]]
    if "reduce_by_key" in s:
        out["reduce_by_key"] = [list(_run_sums(k, v)[:2]) for k, v in zip(*s["reduce_by_key"])]
    return out


def _run_share(kind, mean=16.0):
    """Runs per element: the reciprocal of the mean run length (15,518 for Zipf(1.2) cut at 2^20)."""
    if kind == "geometric":
        return 1.0 / mean
    w = [i ** -1.2 for i in range(1, 1 << 12)]
    tail = lambda e: ((1 << 20) ** e - (1 << 12) ** e) / e  # noqa: E731
    return (sum(w) + tail(-0.2)) / (sum(i * x for i, x in enumerate(w, 1)) + tail(0.8))


def work(case):
    """Bytes: each input read once, each output written once.  One addition a summed element."""
    op = case["op"]
    if op in ("reduce", "scan"):
        return {"bytes": case["n"] * SIZE[case["key"]] * (1 if op == "reduce" else 2), "flops": case["n"]}
    if op in ("merge", "sort"):
        n = case["n"] + case.get("m", 0)
        return {"bytes": 2 * n * (SIZE[case["key"]] + SIZE.get(case["value"], 0)), "flops": 0}
    if op == "reduce_by_key":
        pair = SIZE[case["key"]] + SIZE[case["value"]]
        return {"bytes": case["n"] * pair * (1 + _run_share(case["runs"])), "flops": case["n"]}
    total = {k: sum(ns) for k, ns in _lengths(case).items()}
    return {"bytes": 16 * total.get("sort", 0) + 8 * total.get("scan", 0)
            + 8 * (1 + _run_share("geometric", 32.0)) * total.get("reduce_by_key", 0),
            "flops": total.get("scan", 0) + total.get("reduce_by_key", 0)}
