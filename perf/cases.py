"""Performance cases of the sort library: what a program that uses it has it do.

Every case goes through the public Python entry points of ``sort512cuda``
(``sort``, ``sort_kv``, ``segsort``, ``SegsortPlan``, ``partition``, ``merge``,
``sort_omp_merge``) on seeded synthetic data.  The sorts work in place, so a
pass refills the working array from the kept input and then makes the call.

Sizes and distributions are those of the repository's benchmark and tests
(uniform, normal, lognormal, 256 distinct values, sorted, Zipf(1.1) over 2^20
values, a mixture of 8 Gaussians; lognormal segment lengths), from the smallest
calls to 2^28 doubles.
"""
from __future__ import annotations

import importlib
import math

import torch

s512 = importlib.import_module("avx-512-sort_b200.sort512cuda")

DEVICE = "cuda"
ELEM = {"i32": 4, "f64": 8, "i64": 8, "kv": 8}
TORCH = {"i32": torch.int32, "f64": torch.float64, "i64": torch.int64}
SEG_MAX = 65536  # longest segment of a batch


# ---------------------------------------------------------------------------
# the cases

def listed():
    return [
        # the smallest calls: one short array, all launch and call overhead
        {"name": "sort_i32_tiny", "op": "sort", "dtype": "i32", "n": 777, "dist": "uniform"},
        # an array that one thread block sorts
        {"name": "sort_f64_block", "op": "sort", "dtype": "f64", "n": 10007, "dist": "uniform"},
        # an ordinary array of a million integers
        {"name": "sort_i32_1m", "op": "sort", "dtype": "i32", "n": 1 << 20, "dist": "uniform"},
        # an ordinary array of measurements, odd size
        {"name": "sort_f64_3m", "op": "sort", "dtype": "f64", "n": 3000017, "dist": "normal"},
        # the benchmark's headline size
        {"name": "sort_f64_256m", "op": "sort", "dtype": "f64", "n": 1 << 28, "dist": "uniform"},
        # records by a skewed key: word counts, ids; the value is the row number
        {"name": "sort_kv_zipf", "op": "sort_kv", "dtype": "kv", "n": (1 << 27) + 1, "dist": "zipf"},
        # clustered values with the learned splitters
        {"name": "sort_f64_mix_learned", "op": "sort", "dtype": "f64", "n": 100000007, "dist": "gauss_mix",
         "learned": True},
        # a batch of many uneven arrays, sorted once
        {"name": "segsort_i32_200k", "op": "segsort", "dtype": "i32", "nseg": 200000, "dist": "uniform",
         "plan": False},
        # a batch whose layout stays the same from pass to pass: a captured plan
        {"name": "segsort_f64_plan_50k", "op": "segsort", "dtype": "f64", "nseg": 50000, "dist": "uniform",
         "plan": True},
        # two-way partition around a pivot (a selection step)
        {"name": "partition_f64_20m", "op": "partition", "dtype": "f64", "n": 20000003, "dist": "normal",
         "part": 0.4},
        # two sorted runs into one
        {"name": "merge_f64_32m", "op": "merge", "dtype": "f64", "n": (1 << 25) + 7, "dist": "lognormal",
         "part": 0.37},
        # an array in page-locked host memory, copies included
        {"name": "sort_host_f64_20m", "op": "sort_host", "dtype": "f64", "n": 20000003, "dist": "uniform",
         "pinned": True},
    ]


F64_DISTS = ("uniform", "normal", "lognormal", "distinct256", "ascending", "descending", "gauss_mix")
I32_DISTS = ("uniform", "zipf", "gauss_mix", "ascending")
I64_DISTS = ("uniform", "ascending", "distinct256")


def _dist(rng, dtype):
    return rng.choice(F64_DISTS if dtype == "f64" else I64_DISTS if dtype == "i64" else I32_DISTS)


def _size(rng, lo, hi):
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    op = rng.choice(("sort", "sort", "sort", "sort", "sort_kv", "sort_kv", "segsort", "segsort", "partition", "merge",
                     "sort_omp_merge", "sort_host"))
    if op == "sort":
        dtype = rng.choice(("i32", "f64", "f64", "i64"))
        lo, hi = rng.choice(((2, 16384), (16385, 1 << 24), (1 << 24, 1 << 28)))
        case = {"op": op, "dtype": dtype, "n": _size(rng, lo, hi), "dist": _dist(rng, dtype)}
        if dtype != "i64" and rng.random() < 0.25:
            case["learned"] = True
        return case
    if op == "sort_kv":
        lo, hi = rng.choice(((2, 16384), (16385, 1 << 24), (1 << 24, 1 << 27)))
        return {"op": op, "dtype": "kv", "n": _size(rng, lo, hi), "dist": rng.choice(I32_DISTS)}
    if op == "segsort":
        dtype = rng.choice(("i32", "f64", "kv"))
        return {"op": op, "dtype": dtype, "nseg": _size(rng, 100, 200000),
                "dist": _dist(rng, "i32" if dtype == "kv" else dtype), "plan": rng.random() < 0.5}
    if op == "partition":
        dtype = rng.choice(("i32", "f64", "kv"))
        return {"op": op, "dtype": dtype, "n": _size(rng, 1000, 1 << 26),
                "dist": _dist(rng, "i32" if dtype == "kv" else dtype), "part": round(rng.random(), 3)}
    if op == "merge":
        dtype = rng.choice(("i32", "f64"))
        return {"op": op, "dtype": dtype, "n": _size(rng, 1000, 1 << 26), "dist": _dist(rng, dtype),
                "part": round(rng.random(), 3)}
    if op == "sort_omp_merge":
        dtype = rng.choice(("i32", "f64"))
        return {"op": op, "dtype": dtype, "n": _size(rng, 20000, 1 << 24), "dist": _dist(rng, dtype),
                "parts": rng.choice((2, 5, 8, 16))}
    pinned = rng.random() < 0.7
    dtype = rng.choice(("i32", "f64"))
    return {"op": "sort_host", "dtype": dtype, "n": _size(rng, 10000, 20000003 if pinned else 1 << 21),
            "dist": _dist(rng, dtype), "pinned": pinned}


# ---------------------------------------------------------------------------
# inputs

def _zipf(n, g, s=1.1, ranks=1 << 20):
    w = torch.arange(1, ranks + 1, dtype=torch.float64, device=DEVICE).pow_(-s)
    cdf = torch.cumsum(w, 0)
    cdf /= cdf[-1].clone()
    u = torch.rand(n, dtype=torch.float64, device=DEVICE, generator=g)
    r = torch.searchsorted(cdf, u, right=True).clamp_(max=ranks - 1)
    values = torch.randint(-(1 << 31), 1 << 31, (ranks,), device=DEVICE, generator=g)
    return values[r]


def _gauss_mix(n, g):
    p = torch.rand(16, dtype=torch.float64, device=DEVICE, generator=g)
    means, sigmas = -1e6 + 2e6 * p[:8], 1.0 + 999.0 * p[8:]
    comp = torch.randint(0, 8, (n,), device=DEVICE, generator=g)
    return torch.randn(n, dtype=torch.float64, device=DEVICE, generator=g).mul_(sigmas[comp]).add_(means[comp])


def _values(dtype, dist, n, g):
    """n values of a distribution, on the device."""
    t = TORCH["i32" if dtype == "kv" else dtype]
    if dist == "ascending":
        return torch.sort(_values(dtype, "uniform", n, g)).values
    if dist == "descending":
        return torch.sort(_values(dtype, "uniform", n, g), descending=True).values
    if dist == "distinct256":
        v = _values(dtype, "uniform", 256, g)
        return v[torch.randint(0, 256, (n,), device=DEVICE, generator=g)]
    if dist == "gauss_mix":
        v = _gauss_mix(n, g)
        return v if t.is_floating_point else v.round_().to(t)
    if dist == "zipf":
        return _zipf(n, g).to(t)
    if dtype == "f64":
        if dist == "uniform":
            return torch.rand(n, dtype=t, device=DEVICE, generator=g)
        v = torch.randn(n, dtype=t, device=DEVICE, generator=g)
        return v if dist == "normal" else v.mul_(2.0).exp_()
    if dist != "uniform":
        raise ValueError(f"no distribution {dist} of {dtype}")
    bits = 63 if t == torch.int64 else 31
    return torch.randint(-(1 << bits), (1 << bits) - 1, (n,), dtype=t, device=DEVICE, generator=g)


def _lengths(nseg):
    """Lognormal segment lengths (mu 5, sigma 1.5, within 1..65536): the
    distribution's quantiles, so that a batch of nseg segments always holds
    the same number of keys."""
    q = (torch.arange(nseg, dtype=torch.float64) + 0.5) / nseg
    z = math.sqrt(2.0) * torch.erfinv(2.0 * q - 1.0)
    return torch.exp(5.0 + 1.5 * z).round().clamp(1, SEG_MAX).to(torch.int64)


def _inputs(case, seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    op, dtype, dist = case["op"], case["dtype"], case["dist"]
    got = {}
    if op == "segsort":
        lens = _lengths(case["nseg"]).to(DEVICE)
        lens = lens[torch.randperm(case["nseg"], device=DEVICE, generator=g)]
        got["offsets"] = torch.zeros(case["nseg"] + 1, dtype=torch.int64, device=DEVICE)
        torch.cumsum(lens, 0, out=got["offsets"][1:])
        n = int(got["offsets"][-1])
    else:
        n = case["n"]
    got["keys"] = _values(dtype, dist, n, g)
    if dtype == "kv":
        got["values"] = torch.arange(n, dtype=torch.int32, device=DEVICE)
    if op == "merge":
        got["middle"] = int(case["part"] * n)
        for run in (got["keys"][:got["middle"]], got["keys"][got["middle"]:]):
            run.copy_(torch.sort(run).values)
    if op == "partition":
        # the pivot is an element, at about the asked share of the order
        some = torch.sort(got["keys"][:: max(1, n // 4096)]).values
        got["pivot"] = some[min(some.numel() - 1, int(case["part"] * some.numel()))].item()
    return got


def prepare(case, seed):
    state = _inputs(case, seed)
    state["case"] = case
    state["flags"] = s512.SPLIT_LEARNED if case.get("learned") else 0
    keys = state["keys"]
    if case["op"] == "sort_host":
        state["work"] = torch.empty(keys.numel(), dtype=keys.dtype, pin_memory=case["pinned"])
    else:
        state["work"] = torch.empty_like(keys)
    if "values" in state:
        state["work_values"] = torch.empty_like(state["values"])
    if case.get("plan"):
        dt = {"i32": s512.DTYPE_I32, "f64": s512.DTYPE_F64, "kv": s512.DTYPE_KV_I32}[case["dtype"]]
        state["plan_handle"] = s512.SegsortPlan(dt, state["work"], state["offsets"], values=state.get("work_values"))
    return state


# ---------------------------------------------------------------------------
# one pass

def run(state):
    case, a = state["case"], state["work"]
    a.copy_(state["keys"])
    v = state.get("work_values")
    if v is not None:
        v.copy_(state["values"])
    op = case["op"]
    if op in ("sort", "sort_host"):
        s512.sort(a, flags=state["flags"])
    elif op == "sort_kv":
        s512.sort_kv(a, v)
    elif op == "segsort":
        if case["plan"]:
            state["plan_handle"].launch()
        elif v is not None:
            s512.segsort_kv(a, v, state["offsets"])
        else:
            s512.segsort(a, state["offsets"])
    elif op == "partition":
        n = a.numel()
        if v is not None:
            return {"keys": a, "values": v, "boundary": s512.partition_kv(a, v, 0, n - 1, state["pivot"])}
        return {"keys": a, "boundary": s512.partition(a, 0, n - 1, state["pivot"])}
    elif op == "merge":
        s512.merge(a, state["middle"])
    else:
        s512.sort_omp_merge(a, case["parts"])
    return {"keys": a} if v is None else {"keys": a, "values": v}


def work(case):
    """Every key read once and written once (and a batch's offsets read)."""
    if case["op"] == "segsort":
        n = int(_lengths(case["nseg"]).sum())
        return {"bytes": 2 * n * ELEM[case["dtype"]] + 8 * (case["nseg"] + 1), "flops": 0}
    return {"bytes": 2 * case["n"] * ELEM[case["dtype"]], "flops": 0}


# ---------------------------------------------------------------------------
# the exact results, by torch

def exact(case, seed):
    x = _inputs(case, seed)
    keys, values, op = x["keys"], x.get("values"), case["op"]
    if op == "partition":
        low = keys <= x["pivot"]
        got = {"keys": torch.cat((keys[low], keys[~low].flip(0))), "boundary": int(low.sum())}
        if values is not None:
            got["values"] = torch.cat((values[low], values[~low].flip(0)))
        return got
    if values is not None:  # ordered by key, then value
        order = (keys.to(torch.int64) << 32) + values.to(torch.int64)
    else:
        order = keys
    if op == "segsort":
        nseg = case["nseg"]
        lens = x["offsets"][1:] - x["offsets"][:-1]
        seg = torch.repeat_interleave(torch.arange(nseg, dtype=torch.int32, device=DEVICE), lens)
        order, at = torch.sort(order)
        order = order[torch.sort(seg[at], stable=True).indices]
    else:
        order = torch.sort(order).values
    if values is None:
        return {"keys": order}
    return {"keys": (order >> 32).to(torch.int32), "values": (order & 0xFFFFFFFF).to(torch.int32)}
