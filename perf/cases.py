"""The performance cases of the in-place 213 transpose.

Each case is one call (or one batch) that a program makes through the public
entry points: the plain call, the two decomposition directions, the torch
operators, rank-N permutations and the batched form.  Sizes come from the
configurations, tests and workload generators of this repository, or are
generic; odd and even, small and large, aligned and not.  Every case moves
bytes only, so its floor is one read and one write of the tensor.
"""
from __future__ import annotations

import importlib
import math

import torch

t213 = importlib.import_module("213transpose_b200")
importlib.import_module("213transpose_b200.torch_op")
workloads = importlib.import_module("213transpose_b200.workloads")

# element kinds: torch dtype, elements of that dtype per moved element
KINDS = {
    "u8": (torch.uint8, 1),
    "bf16": (torch.bfloat16, 1),
    "f16": (torch.float16, 1),
    "f32": (torch.float32, 1),
    "i32": (torch.int32, 1),
    "f64": (torch.float64, 1),
    "i64": (torch.int64, 1),
    "b16": (torch.float64, 2),  # 16-byte elements: pairs of doubles
}


def elem_bytes(kind: str) -> int:
    dtype, per = KINDS[kind]
    return torch.empty(0, dtype=dtype).element_size() * per


def listed():
    return [
        # The smallest calls: a few matrices of one layer or one token, where
        # the host path, the launch and one round trip to memory are all.
        {"name": "small", "op": "transpose", "kind": "f32", "d1": 64, "d2": 48, "d3": 4},
        # Many small matrices, the batched transpose of a deep-learning program.
        {"name": "slices", "op": "torch", "kind": "f32", "d1": 512, "d2": 384, "d3": 16},
        # Odd matrices of a few MB, sizes as data gives them.
        {"name": "ragged", "op": "transpose", "kind": "f32", "d1": 1000, "d2": 999, "d3": 4},
        # Half-precision matrices with odd sides: padded vocabularies, ragged sequences.
        {"name": "half_ragged", "op": "torch", "kind": "bf16", "d1": 4099, "d2": 2053, "d3": 8},
        # Large matrices with a large common divisor, the headline configuration.
        {"name": "large", "op": "transpose", "kind": "f32", "d1": 8192, "d2": 6144, "d3": 4},
        # Large coprime matrices in double precision, the second large configuration.
        {"name": "coprime", "op": "transpose", "kind": "f64", "d1": 7919, "d2": 6151, "d3": 2},
        # Array of structures to structure of arrays.
        {"name": "aos", "op": "transpose", "kind": "i32", "d1": 3, "d2": 1 << 22, "d3": 8},
        # Structure of arrays to array of structures, odd counts: long rows, few of them.
        {"name": "soa_ragged", "op": "transpose", "kind": "f32", "d1": 1000003, "d2": 37, "d3": 1},
        # The R2C direction called by name, as programs written for the two halves do.
        {"name": "r2c", "op": "r2c", "kind": "f32", "d1": 3001, "d2": 2000, "d3": 4},
        # Attention heads: (batch, sequence, heads, head size) to (batch, heads, sequence, head size).
        {"name": "heads", "op": "permute", "kind": "f16", "shape": "8,2048,32,128", "dims": "0,2,1,3"},
        # All axes of a rank-4 array reversed (row-major to column-major).
        {"name": "reverse", "op": "permute", "kind": "f32", "shape": "48,60,100,120", "dims": "3,2,1,0"},
        # Uneven tensors of every element size in one batch: a shard of parameters.
        {"name": "batch", "op": "batch", "seed": 1, "count": 64},
    ]


def _log(rng, lo: float, hi: float) -> int:
    return max(1, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    op = rng.choices(["transpose", "torch", "c2r", "r2c", "permute", "batch"], [40, 20, 7, 7, 14, 12])[0]
    if op == "batch":
        return {"op": op, "seed": rng.randrange(1, 10000), "count": _log(rng, 8, 64)}
    kind = rng.choice(["u8", "bf16", "f16", "f32", "f32", "f32", "i32", "f64", "f64", "i64", "b16"])
    total = math.exp(rng.uniform(math.log(5e4), math.log(4e8))) / elem_bytes(kind)
    if op == "permute":
        rank = rng.choice([3, 4, 5])
        # sides about the rank-th root of the volume, each up to three times off
        side = max(2.0, total ** (1.0 / rank))
        shape = [_log(rng, max(2.0, side / 3), side * 3) for _ in range(rank - 1)]
        shape.insert(rng.randrange(rank), max(2, int(total / math.prod(shape))))
        dims = list(range(rank))
        while dims == sorted(dims):
            rng.shuffle(dims)
        return {"op": op, "kind": kind, "shape": ",".join(map(str, shape)), "dims": ",".join(map(str, dims))}
    d3 = rng.choice([1, 1, 2, 4, 8, 16])
    area = max(64.0, total / d3)
    # mostly matrices of moderate aspect, sometimes tall or wide ones
    lo = 2.0 if rng.random() < 0.25 else max(2.0, math.sqrt(area) / 6)
    a = _log(rng, lo, math.sqrt(area))
    b = max(2, int(area / a))
    if rng.random() < 0.4:  # sizes that people choose: multiples of 8
        a, b = max(8, a // 8 * 8), max(8, b // 8 * 8)
    d1, d2 = (a, b) if rng.random() < 0.5 else (b, a)
    return {"op": op, "kind": kind, "d1": d1, "d2": d2, "d3": d3}


def _ints(text: str):
    return [int(v) for v in text.split(",")]


def _values(count: int, kind: str, gen: torch.Generator) -> torch.Tensor:
    dtype, per = KINDS[kind]
    if dtype.is_floating_point:  # uniform in [-1, 1)
        wide = torch.float64 if dtype == torch.float64 else torch.float32
        x = torch.empty(count * per, dtype=wide, device="cuda").uniform_(-1, 1, generator=gen)
        return x.to(dtype)
    info = torch.iinfo(dtype)
    return torch.randint(info.min, info.max, (count * per,), generator=gen, dtype=dtype, device="cuda")


def _batch_shapes(case):
    return workloads.batched_shapes(case["seed"], case["count"])


def _inputs(case, seed: int):
    """The tensors of a case, flat, in the order the case lists them."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["op"] == "batch":
        return [_values(d1 * d2 * d3, kind, gen) for d1, d2, d3, _, kind in _batch_shapes(case)]
    if case["op"] == "permute":
        return [_values(math.prod(_ints(case["shape"])), case["kind"], gen)]
    return [_values(case["d1"] * case["d2"] * case["d3"], case["kind"], gen)]


def prepare(case, seed):
    xs = _inputs(case, seed)
    state = {"case": case, "xs": xs}
    if case["op"] == "batch":
        # the handle a program keeps: planned once, executed many times
        state["batch"] = t213.Batch([(x, d1, d2, d3, eb) for x, (d1, d2, d3, eb, _) in zip(xs, _batch_shapes(case))])
    elif case["op"] == "permute":
        state["shape"], state["dims"] = _ints(case["shape"]), _ints(case["dims"])
    else:
        state["eb"] = elem_bytes(case["kind"])
    return state


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "batch":
        state["batch"].execute()
        return state["xs"]
    x = state["xs"][0]
    if op == "permute":
        if KINDS[case["kind"]][1] == 1:
            return torch.ops.t213.permute_(x.view(state["shape"]), state["dims"])
        n = len(state["dims"])
        t213.permute(x, state["shape"][::-1], [n - 1 - d for d in reversed(state["dims"])], elem_bytes=16)
        return x
    d1, d2, d3 = case["d1"], case["d2"], case["d3"]
    if op == "torch" and KINDS[case["kind"]][1] == 1:
        return torch.ops.t213.transpose_(x.view(d3, d2, d1))
    if op == "c2r":
        t213.inplace.c2r.transpose(x, d1, d2, d3, elem_bytes=state["eb"])
    elif op == "r2c":
        # R2C is given the shape that it makes: the inverse of c2r.transpose(d2, d1)
        t213.inplace.r2c.transpose(x, d2, d1, d3, elem_bytes=state["eb"])
    else:
        t213.inplace.transpose(x, d1, d2, d3, elem_bytes=state["eb"])
    return x


def work(case):
    if case["op"] == "batch":
        nbytes = workloads.total_bytes(_batch_shapes(case))
    elif case["op"] == "permute":
        nbytes = math.prod(_ints(case["shape"])) * elem_bytes(case["kind"])
    else:
        nbytes = case["d1"] * case["d2"] * case["d3"] * elem_bytes(case["kind"])
    return {"bytes": 2 * nbytes, "flops": 0}


def _wide(x: torch.Tensor) -> torch.Tensor:
    return x.double() if x.dtype.is_floating_point else x.long()


def _swapped(x: torch.Tensor, d1: int, d2: int, d3: int, per: int) -> torch.Tensor:
    return x.view(d3, d2, d1, per).transpose(1, 2).contiguous()


def exact(case, seed):
    xs = [_wide(x) for x in _inputs(case, seed)]
    if case["op"] == "batch":
        return [_swapped(x, d1, d2, d3, KINDS[kind][1]).view(-1)
                for x, (d1, d2, d3, _, kind) in zip(xs, _batch_shapes(case))]
    per = KINDS[case["kind"]][1]
    if case["op"] == "permute":
        shape, dims = _ints(case["shape"]), _ints(case["dims"])
        y = xs[0].view(*shape, per).permute(*dims, len(dims)).contiguous()
        return y.squeeze(-1) if per == 1 else y.view(-1)
    y = _swapped(xs[0], case["d1"], case["d2"], case["d3"], per)
    return y.squeeze(-1) if case["op"] == "torch" and per == 1 else y.view(-1)
