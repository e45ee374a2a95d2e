"""What a user of this package has it do, as measurable cases: one call through the public API each.

A case names the operation, the data type, the shape and the distribution of the values.  ``prepare``
makes the device-resident arrays that a program holds before the call, ``run`` makes the call."""
from __future__ import annotations

import math

import numpy as np
import torch

import cupynumeric_b200 as num
from cupynumeric_b200 import workloads

_TORCH = {"int8": torch.int8, "uint8": torch.uint8, "int16": torch.int16, "uint16": torch.uint16,
          "float16": torch.float16, "int32": torch.int32, "uint32": torch.uint32, "float32": torch.float32,
          "int64": torch.int64, "uint64": torch.uint64, "float64": torch.float64,
          "complex64": torch.complex64, "complex128": torch.complex128}
_SIGNED = {torch.uint16: torch.int16, torch.uint32: torch.int32, torch.uint64: torch.int64}


def listed() -> list[dict]:
    return [
        # the smallest calls: a few values ordered inside a larger program, where latency is all there is
        {"name": "sort-small", "op": "sort", "dtype": "int32", "rows": 1, "n": 1000, "values": "full"},
        # an ordinary ranking of a table column of odd length (scores with missing values and ties)
        {"name": "argsort-medium", "op": "argsort", "dtype": "float32", "rows": 1, "n": 100_003, "values": "scores"},
        # the 1-D int32 sort of the benchmark (keys uniform over the full range)
        {"name": "sort-int32-16m", "op": "sort", "dtype": "int32", "rows": 1, "n": 1 << 24, "values": "full"},
        # the benchmark's headline: stable argsort of float32 with NaNs and duplicates, int64 indices
        {"name": "argsort-float32-256m", "op": "argsort", "dtype": "float32", "rows": 1, "n": 1 << 28, "values": "scores"},
        # the benchmark's row sort: many independent rows (per-sample order statistics)
        {"name": "sort-rows-float64", "op": "sort", "dtype": "float64", "rows": 65536, "n": 4096, "values": "unit"},
        # the benchmark's heavily duplicated ids (Zipf, below 2^40)
        {"name": "sort-zipf-256m", "op": "sort", "dtype": "int64", "rows": 1, "n": 1 << 28, "values": "zipf"},
        # the benchmark's almost ordered time stamps, with the permutation wanted
        {"name": "argsort-nearly-sorted-256m", "op": "argsort", "dtype": "uint64", "rows": 1, "n": 1 << 28,
         "values": "nearly_sorted"},
        # ranking the candidates of every query: very many short rows
        {"name": "argsort-short-rows", "op": "argsort", "dtype": "float32", "rows": 250_000, "n": 100, "values": "scores"},
        # every column of a table by itself: axis=0, columns too long for one block
        {"name": "sort-columns", "op": "sort_columns", "dtype": "float32", "rows": 257, "n": 100_003, "values": "scores"},
        # ordering a table by several columns, the last one being the major one
        {"name": "lexsort-table", "op": "lexsort", "dtype": "float64,int32,int16", "rows": 1, "n": 4_000_037,
         "values": "table"},
        # the distinct values of a column of ids
        {"name": "unique-ids", "op": "unique", "dtype": "int64", "rows": 1, "n": 33_554_467, "values": "ids"},
        # looking values up in a sorted table (joins, quantile bins)
        {"name": "searchsorted-left", "op": "searchsorted", "dtype": "float64", "rows": 1, "n": 1 << 24,
         "values": "unit", "queries": 1_000_003, "side": "left"},
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# data type, and how often it is drawn: 4- and 8-byte keys are what most calls see
_DRAWN = ["int32", "float32", "int64", "float64"] * 3 + ["uint32", "uint64", "int16", "uint8", "float16", "uint16", "int8",
                                                         "complex64", "complex128"]


def _values(rng, dtype: str) -> str:
    if dtype.startswith(("float", "complex")):
        return rng.choice(["scores", "scores", "unit"])
    if dtype in ("int64", "uint64"):
        return rng.choice(["full", "zipf", "nearly_sorted"])
    return rng.choice(["full", "few"])


def draw(rng) -> dict:
    op = rng.choice(["sort", "argsort", "rows", "sort_columns", "lexsort", "unique", "searchsorted"])
    dtype = rng.choice(_DRAWN)
    size = _itemsize(dtype)
    if op in ("sort", "argsort"):
        # up to 2^28 keys of at most four bytes, 2^27 of eight
        most = 1 << {1: 28, 2: 28, 4: 28, 8: 27, 16: 24}[size]
        return {"op": op, "dtype": dtype, "rows": 1, "n": _log(rng, 16, most), "values": _values(rng, dtype)}
    if op in ("rows", "sort_columns"):
        if dtype == "complex128":
            dtype, size = "float64", 8
        n = _log(rng, 2, 1 << 17)
        rows = max(1, _log(rng, 1 << 10, 1 << (26 if op == "rows" else 25)) // n)
        values = _values(rng, dtype)
        return {"op": rng.choice(["sort", "argsort"]) if op == "rows" else op, "dtype": dtype, "rows": rows, "n": n,
                "values": "full" if values in ("zipf", "nearly_sorted") else values}
    if op == "lexsort":
        keys = rng.choice(["float64,int32,int16", "int32,int32", "float32,int64", "int64,float64,int32,uint8",
                           "float32,uint16"])
        return {"op": op, "dtype": keys, "rows": 1, "n": _log(rng, 1000, 1 << 24), "values": "table"}
    if op == "unique":
        return {"op": op, "dtype": rng.choice(["int32", "int64", "uint32", "uint64", "float64"]), "rows": 1,
                "n": _log(rng, 1000, 1 << 27), "values": "ids"}
    if dtype == "complex128":
        dtype = "complex64"
    return {"op": op, "dtype": dtype, "rows": 1, "n": _log(rng, 1000, 1 << 26), "values": _values(rng, dtype),
            "queries": _log(rng, 100, 1 << 24), "side": rng.choice(["left", "right"])}


def _itemsize(dtype: str) -> int:
    return np.dtype(dtype).itemsize


def _draw_values(n: int, dtype: str, values: str, gen, seed: int) -> torch.Tensor:
    """n values on the GPU.  full: every bit pattern equally likely; few: a hundred distinct values;
    unit: uniform in [0, 1); scores: normal with 1 % exact duplicates and 0.1 % NaN; ids: n/8 + 1 distinct
    values, a few of them in most places; zipf and nearly_sorted: as the benchmark's workloads draw
    them."""
    t = _TORCH[dtype]
    if values == "zipf":
        return workloads.c4_int64_zipf_shard_device(n, 0, "cuda", seed=seed).view(t)
    if values == "nearly_sorted":
        return workloads.c5_uint64_nearly_sorted_shard_device(n, 0, 1, "cuda", seed=seed).view(t)
    if values == "full":
        raw = torch.randint(0, 256, (n * _itemsize(dtype),), dtype=torch.uint8, device="cuda", generator=gen)
        return raw.view(t)
    if values == "ids":
        k = n // 8 + 1
        names = torch.cumsum(torch.randint(1, 100, (k,), device="cuda", generator=gen), 0)
        more = (torch.rand(n - k, dtype=torch.float64, device="cuda", generator=gen) ** 4 * k).long()
        pick = torch.cat([torch.randperm(k, device="cuda", generator=gen), more])
        return names[pick].to(_SIGNED.get(t, t)).view(t)
    if values == "few":
        return torch.randint(0, 100, (n,), dtype=_SIGNED.get(t, t), device="cuda", generator=gen).view(t)
    if t.is_complex:
        # real parts that repeat, so that the imaginary parts decide
        part = torch.float32 if t == torch.complex64 else torch.float64
        re = torch.randn(n, dtype=part, device="cuda", generator=gen)
        im = torch.randn(n, dtype=part, device="cuda", generator=gen)
        return torch.complex(torch.round(re * 100) / 100, im)
    if values == "unit":
        return torch.rand(n, dtype=t, device="cuda", generator=gen)
    a = torch.randn(n, dtype=t, device="cuda", generator=gen)
    dup = a[50::100]   # (each place written once: the same seed gives the same values)
    if dup.numel():
        dup.copy_(a[torch.randint(0, n, (dup.numel(),), device="cuda", generator=gen)])
    k = n // 1000
    if k:
        a[torch.randint(0, n, (k,), device="cuda", generator=gen)] = float("nan")
    return a


def prepare(case: dict, seed: int) -> dict:
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    op, rows, n = case["op"], case["rows"], case["n"]
    if op == "lexsort":
        # a table's columns: the last key is the major one and has the fewest distinct values
        names, keys = case["dtype"].split(","), []
        for i, d in enumerate(names):
            t = _TORCH[d]
            if i == 0 and t.is_floating_point:
                keys.append(torch.randn(n, dtype=t, device="cuda", generator=gen))
            else:
                top = 100_000 if i == 0 else 200 if i == len(names) - 1 else 3650
                keys.append(torch.randint(0, top, (n,), dtype=torch.int32, device="cuda", generator=gen).to(
                    _SIGNED.get(t, t)).view(t))
        return {"op": op, "keys": [num.array(k) for k in keys]}
    values = _draw_values(rows * n, case["dtype"], case["values"], gen, seed)
    if op == "searchsorted":
        m = case["queries"]
        v = _draw_values(m, case["dtype"], case["values"], gen, seed + 1)
        if case["values"] == "nearly_sorted":
            # look-ups at random places instead of a run at the table's start
            v = torch.randint(0, n, (m,), dtype=torch.int64, device="cuda", generator=gen).view(v.dtype)
        return {"op": op, "a": num.sort(num.array(values)), "v": num.array(v), "side": case["side"]}
    if op == "sort_columns":
        return {"op": op, "a": num.array(values.reshape(n, rows))}
    return {"op": op, "a": num.array(values if rows == 1 else values.reshape(rows, n))}


def run(state: dict):
    op = state["op"]
    if op == "sort":
        out = num.sort(state["a"])
    elif op == "argsort":
        out = num.argsort(state["a"], kind="stable")
    elif op == "sort_columns":
        out = num.sort(state["a"], axis=0)
    elif op == "lexsort":
        out = num.lexsort(state["keys"])
    elif op == "unique":
        out = num.unique(state["a"])
    else:
        out = num.searchsorted(state["a"], state["v"], side=state["side"])
    t = out.torch()
    return t.view(_SIGNED[t.dtype]) if t.dtype in _SIGNED else t   # (the same memory)


def work(case: dict) -> dict:
    """Every input read once and every output written once."""
    total = case["rows"] * case["n"]
    read = sum(_itemsize(d) for d in case["dtype"].split(",")) * total
    op = case["op"]
    if op in ("sort", "sort_columns"):
        return {"bytes": 2 * read, "flops": 0}
    if op in ("argsort", "lexsort"):
        return {"bytes": read + 8 * total, "flops": 0}
    if op == "unique":
        return {"bytes": read + (total // 8 + 1) * _itemsize(case["dtype"]), "flops": 0}
    return {"bytes": read + (_itemsize(case["dtype"]) + 8) * case["queries"], "flops": 0}


def tolerance(case: dict):
    """Sorting moves values and computes none: every output is determined to the bit."""
    return "exact"
