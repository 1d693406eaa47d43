"""Performance cases: the work a program has this library do, through the public Python entry points.

A case is one algorithm call on device-resident data: operation, number of elements, element types
and the options that change what the kernels do.  Sizes go from the small calls inside an iterative
solver or a per-frame loop, where a call is launches and latency, up to the 2^28-element arrays of the
benchmark.  Types are the 4- and 8-byte ones; inputs follow the value ranges of the benchmark's
workloads (thrust_b200/datagen.py), made on the GPU from the seed.

    listed()            the cases by name
    draw(rng)           one more case of the same ranges
    prepare(case, seed) device inputs and, for the in-place algorithms, the buffer they work in
    run(state)          one call, and everything it produced
    work(case)          bytes that any implementation reads and writes: every input and output once
    tolerance(case)     how far two correct results may be apart
    exact(case, seed)   the floating-point sums as torch gives them without rounding error, for the cases that have any

The in-place algorithms (sort, sort_by_key, stable_sort_zip, partition) overwrite their input, so a
pass copies the input into the work buffer first, as a program does that still needs the original.
"""
import math

import numpy as np
import torch

import thrust_b200 as tb

DTYPES = {"i32": torch.int32, "u32": torch.uint32, "i64": torch.int64, "u64": torch.uint64, "f32": torch.float32, "f64": torch.float64}
SIZE = {"i32": 4, "u32": 4, "i64": 8, "u64": 8, "f32": 4, "f64": 8}
SIGNED = {"u32": torch.int32, "u64": torch.int64}     # the torch type the values are drawn in and handed back as
NUMPY = {"i32": np.int32, "u32": np.uint32, "i64": np.int64, "u64": np.uint64, "f32": np.float32, "f64": np.float64}

#: Largest n that draw() takes, per operation: at most the time of the largest listed case.
LARGEST = {"reduce": 1 << 28, "inclusive_scan": 1 << 28, "exclusive_scan": 1 << 28, "sort": 1 << 27, "sort_by_key": 1 << 26, "copy_if": 1 << 28,
           "partition": 1 << 28, "unique": 1 << 28, "reduce_by_key": 1 << 28, "merge_by_key": 1 << 27, "stable_sort_zip": 1 << 25}
SMALLEST = 1000


def listed():
    return [
        # the norm, residual or count of a small vector inside a solver's loop: one number wanted now
        {"name": "reduce_i32_1k", "op": "reduce", "n": 1000, "type": "i32", "acc": "i64", "fold": "plus"},
        # offsets of a short list of row lengths (CSR row pointers, output slots of a frame)
        {"name": "scan_i32_50k", "op": "inclusive_scan", "n": 50001, "type": "i32", "fold": "plus"},
        # ranking a batch of scores or distances; keys only
        {"name": "sort_f32_100k", "op": "sort", "n": 100003, "type": "f32", "descending": False, "distinct": 0},
        # keeping the records that pass a filter, an ordinary batch
        {"name": "copy_if_i32_1m", "op": "copy_if", "n": 1000003, "type": "i32", "keep": 0.5},
        # grouped sums after a sort (histogram, sparse assembly); runs of mean length 4
        {"name": "reduce_by_key_i32_f32_5m", "op": "reduce_by_key", "n": 5000011, "type": "i32", "value": "f32", "run": 4},
        # (Morton code or packed id, index) pairs: 64-bit keys of which 40 bits vary
        {"name": "sort_by_key_u64_u32_20m", "op": "sort_by_key", "n": 20000003, "type": "u64", "value": "u32", "descending": False, "distinct": 0},
        # stable sort of zipped records under a comparator, the comparison-sort route
        {"name": "stable_sort_zip_u32_f32_8m", "op": "stable_sort_zip", "n": 8000009, "type": "u32", "value": "f32"},
        # joining two sorted tables, the shape of the benchmark's merge at half its size
        {"name": "merge_by_key_u64_u32_2p27", "op": "merge_by_key", "n": 1 << 27, "type": "u64", "value": "u32", "share": 0.5},
        # splitting a large array in place by a flag
        {"name": "partition_i32_2p27", "op": "partition", "n": 1 << 27, "type": "i32", "keep": 0.5},
        # the benchmark's headline sizes: whole-array sum, prefix sum and sort
        {"name": "reduce_i32_2p28", "op": "reduce", "n": 1 << 28, "type": "i32", "acc": "i64", "fold": "plus"},
        {"name": "scan_f32_2p28", "op": "exclusive_scan", "n": 1 << 28, "type": "f32", "fold": "plus"},
        {"name": "sort_by_key_u32_u32_2p28", "op": "sort_by_key", "n": 1 << 28, "type": "u32", "value": "u32", "descending": False, "distinct": 0},
    ]


def draw(rng):
    op = rng.choice(sorted(LARGEST))
    n = int(math.exp(rng.uniform(math.log(SMALLEST), math.log(LARGEST[op]))))
    case = {"op": op, "n": n}
    if op in ("reduce", "inclusive_scan", "exclusive_scan"):
        case["type"] = rng.choice(["i32", "i32", "f32", "f32", "i64", "f64"])
        case["fold"] = rng.choice(["plus", "plus", "plus", "min", "max"])
        if op == "reduce":
            case["acc"] = "i64" if case["type"] == "i32" and case["fold"] == "plus" else case["type"]
    elif op in ("sort", "sort_by_key"):
        case["type"] = rng.choice(["u32", "i32", "f32", "u64", "i64", "f64"])
        case["descending"] = rng.random() < 0.25
        case["distinct"] = 0 if rng.random() < 0.7 else int(10 ** rng.uniform(2, 6))
        if op == "sort_by_key":
            case["value"] = rng.choice(["u32", "u32", "i64"])
    elif op in ("copy_if", "partition"):
        case["type"] = rng.choice(["i32", "i32", "f32", "i64"])
        case["keep"] = rng.choice([0.02, 0.25, 0.5, 0.5, 0.9])
    elif op == "unique":
        case["type"] = rng.choice(["i32", "i32", "i64"])
        case["run"] = rng.choice([1.25, 4, 30])
    elif op == "reduce_by_key":
        case["type"] = rng.choice(["i32", "i32", "i64"])
        case["value"] = rng.choice(["f32", "i32", "f64"])
        case["run"] = rng.choice([1.25, 4, 30])
    elif op == "merge_by_key":
        case["type"] = rng.choice(["u64", "u32", "i32", "f32"])
        case["value"] = rng.choice(["u32", "u32", "none"])
        case["share"] = rng.choice([0.5, 0.5, 0.9])
    else:
        case["type"] = rng.choice(["u32", "i32", "f32"])
        case["value"] = "f32"
    if op not in ("reduce", "stable_sort_zip", "sort") and SIZE[case["type"]] + SIZE.get(case.get("value", "none"), 0) > 8:
        case["n"] = min(case["n"], LARGEST[op] // 2 + 1)
    if op == "sort" and SIZE[case["type"]] == 8:
        case["n"] = min(case["n"], LARGEST[op] // 4 + 1)
    return case


# ------------------------------------------------------------------------------------- inputs
def _typed(x, name):
    """x's values (already in range) as a tensor of the named type."""
    if name in SIGNED:
        return x.to(SIGNED[name]).view(DTYPES[name])
    return x.to(DTYPES[name])


def _keys(g, n, name, distinct):
    """Sort keys: all bits random, a limited number of distinct values, or 40 random bits for u64 (packed
    ids); floats are normally distributed."""
    if distinct:
        return _typed(torch.randint(0, distinct, (n,), generator=g, device="cuda", dtype=torch.int32), name)
    if name in ("f32", "f64"):
        return torch.randn(n, generator=g, device="cuda", dtype=DTYPES[name])
    if name == "u64":
        return _typed(torch.randint(0, 1 << 40, (n,), generator=g, device="cuda", dtype=torch.int64), name)
    wide = torch.int64 if name == "i64" else torch.int32
    lo, hi = (-(1 << 62), 1 << 62) if name == "i64" else (-(1 << 31), (1 << 31) - 1)
    return _typed(torch.randint(lo, hi, (n,), generator=g, device="cuda", dtype=wide), name)


def runs_of(case):
    return max(1, int(case["n"] / case["run"]))


def _run_keys(g, n, name, mean, runs):
    """Sorted keys in `runs` runs of nearly geometric length with the given mean, consecutive keys 1 to 8
    apart.  A few too many positions are drawn as run starts and the surplus is taken out at even steps."""
    p = 1.0 / mean
    heads = torch.rand(n, generator=g, device="cuda") < min(1.0, p + 6.0 * math.sqrt(p / n))
    heads[0] = True
    starts = torch.nonzero(heads).view(-1)
    surplus = starts.numel() - runs
    if surplus > 0:
        heads[starts[1 + torch.arange(surplus, device="cuda") * (starts.numel() - 1) // surplus]] = False
    gaps = torch.randint(1, 9, (n,), generator=g, device="cuda", dtype=torch.int32)
    return _typed(torch.cumsum(gaps * heads, 0, dtype=torch.int64), name)


def _sorted_keys(g, n, name):
    if name == "f32":
        return torch.sort(torch.randn(n, generator=g, device="cuda"))[0]
    if name == "i32":
        return torch.sort(torch.randint(-(1 << 31), (1 << 31) - 1, (n,), generator=g, device="cuda", dtype=torch.int32))[0]
    wide = torch.randint(0, 1 << (48 if name == "u64" else 32), (n,), generator=g, device="cuda", dtype=torch.int64)
    return _typed(torch.sort(wide)[0], name)


def _values(g, n, name):
    """Payloads: an index (u32, i64), or numbers to add up."""
    if name in ("f32", "f64"):
        return torch.rand(n, generator=g, device="cuda", dtype=DTYPES[name])
    if name == "i32":
        return torch.randint(-1000, 1000, (n,), generator=g, device="cuda", dtype=torch.int32)
    return _typed(torch.arange(n, device="cuda", dtype=torch.int64 if name == "i64" else torch.int32), name)


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    op, n, t = case["op"], case["n"], case["type"]
    s = dict(case)
    if op in ("reduce", "inclusive_scan", "exclusive_scan"):
        if t in ("f32", "f64"):
            s["x"] = torch.rand(n, generator=g, device="cuda", dtype=DTYPES[t])
        else:
            lo, hi = (-(1 << 20), 1 << 20) if op == "reduce" else (0, 16)
            s["x"] = torch.randint(lo, hi, (n,), generator=g, device="cuda", dtype=DTYPES[t])
        if op == "reduce":      # the identity of the fold, in the accumulator's type
            acc = NUMPY[case["acc"]]
            ends = np.finfo(acc) if case["acc"] in ("f32", "f64") else np.iinfo(acc)
            s["init"] = acc({"plus": 0, "min": ends.max, "max": ends.min}[case["fold"]])
    elif op in ("sort", "sort_by_key", "stable_sort_zip"):
        s["keys"] = _keys(g, n, t, case.get("distinct", 0))
        s["keys_work"] = torch.empty_like(s["keys"])
        if op != "sort":
            s["vals"] = _values(g, n, case["value"])
            s["vals_work"] = torch.empty_like(s["vals"])
    elif op in ("copy_if", "partition"):
        span = 1 << 31
        x = torch.randint(0, span - 1, (n,), generator=g, device="cuda", dtype=torch.int32)
        s["x"] = _typed(x, t)
        s["pred"] = ("mod_eq", 2, 0) if case["keep"] == 0.5 and t != "f32" else ("lt", int(case["keep"] * span), 0)
        s["work" if op == "partition" else "out"] = torch.zeros_like(s["x"])
    elif op == "unique":
        s["x"] = _run_keys(g, n, t, case["run"], runs_of(case))
    elif op == "reduce_by_key":
        s["keys"] = _run_keys(g, n, t, case["run"], runs_of(case))
        s["vals"] = _values(g, n, case["value"])
    elif op == "merge_by_key":
        na = int(n * case["share"])
        s["a"], s["b"] = _sorted_keys(g, na, t), _sorted_keys(g, n - na, t)
        s["va"], s["vb"] = None, None
        if case["value"] != "none":
            s["va"], s["vb"] = _values(g, na, case["value"]), _values(g, n - na, case["value"])
    return s


# ------------------------------------------------------------------------------------- one pass
def _plain(t):
    """A tensor of an unsigned type as the signed type of its size: the same bits, no copy."""
    return t.view(torch.int32) if t.dtype == torch.uint32 else t.view(torch.int64) if t.dtype == torch.uint64 else t


def run(s):
    op = s["op"]
    if op == "reduce":
        return tb.reduce(s["x"], s["init"], op=s["fold"])
    if op == "inclusive_scan":
        return tb.inclusive_scan(s["x"], op=s["fold"])
    if op == "exclusive_scan":
        return tb.exclusive_scan(s["x"], 0, op=s["fold"])
    if op == "sort":
        s["keys_work"].copy_(s["keys"])
        return _plain(tb.sort(s["keys_work"], descending=s["descending"]))
    if op == "sort_by_key":
        s["keys_work"].copy_(s["keys"])
        s["vals_work"].copy_(s["vals"])
        k, v = tb.sort_by_key(s["keys_work"], s["vals_work"], descending=s["descending"])
        return _plain(k), _plain(v)
    if op == "stable_sort_zip":
        s["keys_work"].copy_(s["keys"])
        s["vals_work"].copy_(s["vals"])
        k, v = tb.stable_sort_zip_by_first(s["keys_work"], s["vals_work"])
        return _plain(k), _plain(v)
    if op == "copy_if":
        return tb.copy_if(s["x"], *s["pred"], out=s["out"]).numel(), s["out"]
    if op == "partition":
        s["work"].copy_(s["x"])
        return tb.partition(s["work"], *s["pred"]), s["work"]
    if op == "unique":
        return tb.unique_copy(s["x"])
    if op == "reduce_by_key":
        return tb.reduce_by_key(s["keys"], s["vals"])
    k, v = tb.merge_by_key(s["a"], s["b"], s["va"], s["vb"])
    return _plain(k) if v is None else (_plain(k), _plain(v))


# ------------------------------------------------------------------------------------- bounds
def work(case):
    op, n = case["op"], case["n"]
    record = SIZE[case["type"]] + SIZE.get(case.get("value", "none"), 0)
    kept = {"reduce": 0.0, "copy_if": case.get("keep", 0), "unique": 1.0 / case.get("run", 1), "reduce_by_key": 1.0 / case.get("run", 1)}.get(op, 1.0)
    return {"bytes": n * record * (1.0 + kept) + 8, "flops": 0}


def tolerance(case):
    """Whole numbers, copies and orders are exact.  Sums of floats depend on how they are associated:
    the figures are about four times what the library's sums differ by from sums in twice the precision."""
    summed = _summed(case)
    if summed is None:
        return "exact"
    return {"rel": 2e-6, "max": 1e-5} if summed == "f32" else {"rel": 1e-14, "max": 1e-13}


def _summed(case):
    """The type in which the case adds floats up, or None."""
    t = case.get("value") if case["op"] == "reduce_by_key" else case["type"] if case["op"] in ("reduce", "inclusive_scan", "exclusive_scan") else None
    return t if t in ("f32", "f64") and case.get("fold", "plus") == "plus" else None


def _prefix_sums(x):
    """Inclusive prefix sums of x, whose values lie in [0, 1) on torch.rand's grid (multiples of 2^-24, or of 2^-53
    for doubles): added up in whole numbers, so that the only rounding is that of the result to 64 bits."""
    if x.dtype == torch.float32:
        return torch.cumsum((x.double() * 2.0 ** 24).long(), 0).double() * 2.0 ** -24
    scaled = (x * 2.0 ** 53).long()
    high, low = torch.cumsum(scaled >> 27, 0), torch.cumsum(scaled & ((1 << 27) - 1), 0)
    return high.double() * 2.0 ** -26 + low.double() * 2.0 ** -53


def exact(case, seed):
    """What run() returns, its float sums free of rounding errors; None where nothing is added up in floats
    (those outputs are whole numbers and copies, which are compared exactly)."""
    if _summed(case) is None:
        return None
    s = prepare(case, seed)
    if case["op"] == "reduce":
        return float(_prefix_sums(s["x"])[-1])
    if case["op"] == "inclusive_scan":
        return _prefix_sums(s["x"])
    if case["op"] == "exclusive_scan":
        return torch.cat([torch.zeros(1, dtype=torch.float64, device="cuda"), _prefix_sums(s["x"])[:-1]])
    _, lengths = torch.unique_consecutive(s["keys"], return_counts=True)
    ends = _prefix_sums(s["vals"])[torch.cumsum(lengths, 0) - 1]
    return None, torch.diff(ends, prepend=torch.zeros(1, dtype=torch.float64, device="cuda"))
