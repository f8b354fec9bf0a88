"""Workloads that stand for what this package is used for, with the bytes they cannot do without.

``listed()`` names them, ``draw(rng)`` gives further ones from the same ranges, ``prepare`` builds what a program holds
before the call, ``run`` is one pass through the public entry points (``IntNBitTableBatchedEmbeddingBags``,
``PermutePooledEmbeddings`` and the ``torch.ops.fbgemm`` operators).
"""
from __future__ import annotations

import math

import torch

import fbgemm_ascend_b200 as fa
from fbgemm_ascend_b200.types import row_bytes
from fbgemm_ascend_b200.workloads import WorkloadSpec, build_tables

TYPES = {"int8": fa.SparseType.INT8, "int4": fa.SparseType.INT4, "int2": fa.SparseType.INT2, "fp16": fa.SparseType.FP16,
         "fp8": fa.SparseType.FP8, "fp32": fa.SparseType.FP32}
OUTPUTS = {"fp32": fa.SparseType.FP32, "fp16": fa.SparseType.FP16, "bf16": fa.SparseType.BF16}
DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}
SIZES = {"fp32": 4, "fp16": 2, "bf16": 2}
POOLINGS = {"sum": fa.PoolingMode.SUM, "mean": fa.PoolingMode.MEAN, "none": fa.PoolingMode.NONE}


def _lookup(name, tables, rows, dims, types, batch, lengths, indices, bits, pooling, output, weighted=False, pruned=0.0):
    """A lookup; ``dims`` and ``types`` are repeated over the tables, ``lengths`` and ``indices`` are the distributions of
    the bags and of the rows they name (see WorkloadSpec), ``pruned`` the share of indices that are -1."""
    return {"name": name, "kind": "lookup", "tables": tables, "rows": rows, "dims": dims, "types": types, "batch": batch,
            "lengths": lengths, "indices": indices, "bits": bits, "pooling": pooling, "output": output, "weighted": weighted,
            "pruned": pruned}


def listed():
    return [
        # One table, one small request: the smallest call a ranking service makes; launch and host time are what count.
        _lookup("one_table", 1, 100_000, "128", "int8", 512, "fixed:20", "uniform", 32, "sum", "fp16"),
        # A whole small request from its arrival: jagged features put into table order, lengths to offsets, lookup, pooled
        # rows into feature order.
        {"name": "small_request", "kind": "request", "tables": 26, "rows": 200_000, "dims": "128", "types": "int8", "batch": 64,
         "lengths": "poisson:30:1:100", "indices": "zipf:1.05", "bits": 64, "pooling": "sum", "output": "fp16"},
        # An ordinary recommendation request: 26 tables of a million rows, hot rows looked up again and again.
        _lookup("serving", 26, 1_000_000, "128", "int8", 2048, "poisson:30:1:100", "zipf:1.05", 64, "sum", "fp16"),
        # The largest: one rank's shard of a table-wise sharded model over the global batch (3M of the 12M rows per table,
        # so that a state fits the card several times).
        _lookup("shard_step", 64, 3_000_000, "128", "int8", 65536, "poisson:32:1:128", "zipf:1.05", 64, "sum", "fp16"),
        # Compressed tables of several widths, mean pooling, 32-bit indices, full-precision result.
        _lookup("int4_widths_mean", 64, 2_500_000, "64,128,256", "int4", 16384, "fixed:40", "zipf:1.1", 32, "mean", "fp32"),
        # Weighted pooling over tables of different types, long ragged bags, no locality.
        _lookup("weighted_types", 96, 1_000_000, "128", "int8,int4,fp16", 8192, "uniform:0:200", "uniform", 64, "sum", "fp32", True),
        # A model that grew over time: odd and wide tables of four types, empty bags, pruned rows, an odd batch.
        _lookup("ragged_tables", 16, 200_000, "36,48,200,96,1024,256,20,512", "int8,int4,fp16,fp8", 777, "uniform:0:100", "zipf:1.05", 32,
                "mean", "bf16", False, 0.02),
        # Sequence features, cut and padded to one length: every row comes back by itself.
        _lookup("sequence", 26, 1_000_000, "128", "int8", 2048, "fixed:30", "zipf:1.05", 64, "none", "fp16"),
        # A request of a large batch put into table order, and its offsets (what stands in front of a sharded lookup).
        {"name": "input_order", "kind": "input", "tables": 64, "batch": 16384, "lengths": "poisson:32:1:128", "bits": 64, "weighted": False},
        # Pooled rows put into feature order, and the gradient back: what a model over these tables does in training.
        {"name": "feature_order", "kind": "order", "tables": 512, "dims": "128", "batch": 8192, "dtype": "fp16", "backward": True},
        # Publishing a trained table: fp32 rows to 8-bit rows.
        {"name": "quantize", "kind": "rowwise", "op": "quantize8", "rows": 1_000_000, "cols": 128},
        # Reading a compressed table back as fp32.
        {"name": "dequantize", "kind": "rowwise", "op": "dequantize4", "rows": 1_000_000, "cols": 128},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _lengths(rng):
    mean = _log(rng, 3, 100)
    return mean, rng.choice(["fixed:%d" % mean, "poisson:%d:1:%d" % (mean, 4 * mean), "uniform:0:%d" % (2 * mean)])


def _dims(rng, types):
    """A width for every entry of ``types``: mostly 64, 128 or 256, sometimes anything up to 1024 that the types take."""
    step = 8 if "int4" in types else 4
    n = len(types.split(","))
    if rng.random() < 0.7:
        return ",".join(str(rng.choice([32, 64, 128, 128, 256])) for _ in range(n))
    return ",".join(str(max(step, _log(rng, 16, 1024) // step * step)) for _ in range(n))


def _draw_lookup(rng):
    types = rng.choice(["int8", "int8", "int8", "int4", "fp16", "fp8", "int8,int4,fp16"])
    pooling = rng.choice(["sum", "sum", "mean", "none"])
    if pooling == "none":
        dims = str(rng.choice([32, 64, 96, 128, 256]))
        types = rng.choice(["int8", "int8", "int4", "fp16"])
    else:
        dims = _dims(rng, types)
    mean, lengths = _lengths(rng)
    if pooling == "none":
        lengths = "fixed:%d" % mean
    bits = rng.choice([32, 64])
    output = rng.choice(["fp16", "fp16", "fp32", "bf16"])
    weighted = pooling != "none" and rng.random() < 0.3
    widest = max(int(d) for d in dims.split(","))
    tables = _log(rng, 1, 96)
    batch = _log(rng, 8, 65536)
    # neither more rows per pass, nor larger tables and results, than a fifth of the largest listed case
    batch = max(1, min(batch, 26_000_000 * 128 // (tables * mean * max(widest, 128)), 200_000_000 // (tables * widest)))
    if pooling == "none":
        batch = max(1, min(batch, 400_000_000 // (tables * mean * widest)))
    rows = max(100, min(_log(rng, 1000, 3_000_000), 5_000_000_000 // (tables * (2 * widest + 16))))
    indices = rng.choice(["zipf:1.05", "zipf:1.1", "uniform"])
    c = _lookup("", tables, rows, dims, types, batch, lengths, indices, bits, pooling, output, weighted, rng.choice([0.0, 0.0, 0.02]))
    del c["name"]
    return c


def draw(rng):
    kind = rng.choice(["lookup"] * 7 + ["request", "request", "input", "order", "rowwise", "rowwise"])
    if kind == "lookup":
        return _draw_lookup(rng)
    if kind == "request":
        return {"kind": "request", "tables": _log(rng, 2, 64), "rows": _log(rng, 10_000, 500_000), "dims": rng.choice(["64", "128", "64,128"]),
                "types": rng.choice(["int8", "int8", "int4", "fp16"]), "batch": _log(rng, 8, 1024), "lengths": _lengths(rng)[1],
                "indices": "zipf:1.05", "bits": rng.choice([32, 64]), "pooling": rng.choice(["sum", "mean"]),
                "output": rng.choice(["fp16", "fp32"])}
    if kind == "input":
        tables = _log(rng, 4, 256)
        mean, lengths = _lengths(rng)
        return {"kind": "input", "tables": tables, "batch": max(1, min(_log(rng, 64, 65536), 50_000_000 // (tables * mean))), "lengths": lengths,
                "bits": rng.choice([32, 64]), "weighted": rng.random() < 0.4}
    if kind == "order":
        tables = _log(rng, 4, 512)
        dims = rng.choice(["128", "64,128,256", "20,36,100"])
        widest = max(int(d) for d in dims.split(","))
        return {"kind": "order", "tables": tables, "dims": dims, "batch": max(1, min(_log(rng, 64, 16384), 400_000_000 // (tables * widest))),
                "dtype": rng.choice(["fp16", "fp32", "bf16"]), "backward": rng.random() < 0.5}
    cols = rng.choice([32, 64, 128, 128, 256, 4 * _log(rng, 4, 256)])
    op = rng.choice(["quantize8", "dequantize8", "quantize4", "dequantize4", "table8", "table4"])
    if op[-1] == "4":
        cols = cols // 8 * 8
    return {"kind": "rowwise", "op": op, "rows": _log(rng, 1000, 400_000_000 // cols), "cols": cols}


# ---- what a case is made of ---------------------------------------------------------------------------

def _spec(case, seed):
    n = case["tables"]
    dims = [int(d) for d in case["dims"].split(",")]
    types = [TYPES[t] for t in case["types"].split(",")]
    return WorkloadSpec(case.get("name") or "drawn", n, case["rows"], [dims[t % len(dims)] for t in range(n)],
                        [types[t % len(types)] for t in range(n)], case["batch"], POOLINGS[case["pooling"]], OUTPUTS[case["output"]],
                        torch.int32 if case["bits"] == 32 else torch.int64, case["lengths"], case["indices"],
                        case.get("weighted", False), "normal:0.05", int(seed))


def _random_lengths(dist, n, gen, device):
    """Lengths of the distribution, a few of them one more or less so that every seed's sum is the same."""
    kind, *v = dist.split(":")
    if kind == "fixed":
        return torch.full((n,), int(v[0]), dtype=torch.int64, device=device)
    if kind == "poisson":
        lengths = torch.poisson(torch.full((n,), float(v[0]), device=device), generator=gen).to(torch.int64).clamp_(int(v[1]), int(v[2]))
    else:
        lengths = torch.randint(int(v[0]), int(v[1]) + 1, (n,), generator=gen, device=device)
    while (off := round(n * _mean_length(dist)) - int(lengths.sum())) != 0:
        some = torch.randperm(n, generator=gen, device=device)[: abs(off)]
        lengths[some] = (lengths[some] + (1 if off > 0 else -1)).clamp_(min=0)
    return lengths


def _mean_length(dist):
    kind, *v = dist.split(":")
    return (int(v[0]) + int(v[1])) / 2 if kind == "uniform" else float(v[0])


def _order_module(dims, gen, device):
    """Features in a random order, as a model's own order is to its tables'."""
    order = torch.randperm(len(dims), generator=gen, device=device).tolist()
    return fa.PermutePooledEmbeddings(dims, order, device=device)


def _rows_of(dist, rows, n, gen, device):
    """n row numbers of a table: uniform, or bounded power law ("zipf:exponent") with the hot rows scattered over the table."""
    if dist == "uniform":
        return torch.randint(0, rows, (n,), generator=gen, device=device)
    a = 1.0 - float(dist.split(":")[1])
    u = torch.rand(n, generator=gen, device=device, dtype=torch.float64)
    rank = (1.0 + u * ((rows + 1.0) ** a - 1.0)).pow_(1.0 / a).to(torch.int64).clamp_(1, rows) - 1
    return torch.randperm(rows, generator=gen, device=device)[rank]


def _batch(ws, gen, device):
    """A request in table order: indices, offsets [T * B + 1], per-sample weights or None."""
    lengths = _random_lengths(ws.length_dist, ws.T * ws.B, gen, device)
    per_table = lengths.view(ws.T, ws.B).sum(1).tolist()
    indices = torch.cat([_rows_of(ws.index_dist, ws.E, n, gen, device).to(ws.index_dtype) for n in per_table])
    offsets = torch.zeros(ws.T * ws.B + 1, dtype=torch.int64, device=device)
    offsets[1:] = torch.cumsum(lengths, 0)
    weights = torch.rand(indices.numel(), generator=gen, device=device) if ws.weighted else None
    return indices, offsets.to(ws.index_dtype), weights


def _in_feature_order(indices, offsets, tables, gen, device):
    """A request in table order as it arrives: features in an order of their own (lengths and indices), and the permute
    list that brings it into table order."""
    permute = torch.randperm(tables, generator=gen, device=device)
    lengths = (offsets[1:] - offsets[:-1]).view(tables, -1)
    starts = offsets[:: lengths.shape[1]].tolist()
    arrival = torch.argsort(permute).tolist()       # input feature j is table arrival[j]: output table i is input permute[i]
    values = torch.cat([indices[starts[t]:starts[t + 1]] for t in arrival])
    return permute.to(torch.int32), lengths[torch.tensor(arrival, device=device)].contiguous(), values


def prepare(case, seed):
    device = torch.device("cuda")
    gen = torch.Generator(device=device)
    gen.manual_seed(int(seed) * 2 + 1)
    kind = case["kind"]
    s = {"kind": kind}
    if kind in ("lookup", "request"):
        ws = _spec(case, seed)
        s["tables"] = build_tables(ws, device)
        indices, offsets, s["weights"] = _batch(ws, gen, device)
        if kind == "request":
            s["permute"], s["lengths"], s["values"] = _in_feature_order(indices, offsets, ws.T, gen, device)
            s["total"] = indices.numel()
            s["order"] = _order_module(ws.dims, gen, device)
            return s
        if case["pruned"] > 0:
            indices.masked_fill_(torch.rand(indices.numel(), generator=gen, device=device) < case["pruned"], -1)
        s["indices"], s["offsets"] = indices, offsets
    elif kind == "input":
        dtype = torch.int32 if case["bits"] == 32 else torch.int64
        n = case["tables"] * case["batch"]
        lengths = _random_lengths(case["lengths"], n, gen, device)
        s["total"] = int(lengths.sum())
        s["lengths"] = lengths.to(dtype).view(case["tables"], case["batch"])
        s["permute"] = torch.randperm(case["tables"], generator=gen, device=device).to(torch.int32)
        s["values"] = torch.randint(0, 3_000_000, (s["total"],), generator=gen, device=device, dtype=dtype)
        s["weights"] = torch.rand(s["total"], generator=gen, device=device) if case["weighted"] else None
    elif kind == "order":
        dims = [int(d) for d in case["dims"].split(",")]
        dims = [dims[t % len(dims)] for t in range(case["tables"])]
        dtype = DTYPES[case["dtype"]]
        s["order"] = _order_module(dims, gen, device)
        s["pooled"] = torch.randn(case["batch"], sum(dims), generator=gen, device=device, dtype=dtype)
        s["grad"] = torch.randn(case["batch"], sum(dims), generator=gen, device=device, dtype=dtype) if case["backward"] else None
        s["pooled"].requires_grad_(case["backward"])
    else:
        x = torch.randn(case["rows"], case["cols"], generator=gen, device=device) * 0.05
        s["op"] = op = case["op"]
        if op == "dequantize8":
            x = torch.ops.fbgemm.FloatToFused8BitRowwiseQuantized(x)
        elif op == "dequantize4":
            x = torch.ops.fbgemm.FloatToFusedNBitRowwiseQuantizedSBHalf(x, 4)
        elif op.startswith("table"):
            s["tables"] = fa.IntNBitTableBatchedEmbeddingBags([("t", case["rows"], case["cols"], TYPES["int" + op[-1]])], device=device)
        s["x"] = x
    return s


def run(s):
    ops = torch.ops.fbgemm
    kind = s["kind"]
    if kind == "lookup":
        return s["tables"](s["indices"], s["offsets"], s["weights"])
    if kind == "request":
        lengths, indices, _ = ops.permute_2D_sparse_data(s["permute"], s["lengths"], s["values"], None, s["total"])
        offsets = ops.asynchronous_complete_cumsum(lengths.view(-1))
        return s["order"](s["tables"](indices, offsets))
    if kind == "input":
        lengths, values, weights = ops.permute_2D_sparse_data(s["permute"], s["lengths"], s["values"], s["weights"], s["total"])
        return lengths, values, weights, ops.asynchronous_complete_cumsum(lengths.view(-1))
    if kind == "order":
        out = s["order"](s["pooled"])
        return (out,) if s["grad"] is None else (out, torch.autograd.grad(out, s["pooled"], s["grad"])[0])
    x, op = s["x"], s["op"]
    if op == "quantize8":
        return ops.FloatToFused8BitRowwiseQuantized(x)
    if op == "quantize4":
        return ops.FloatToFusedNBitRowwiseQuantizedSBHalf(x, 4)
    if op == "dequantize8":
        return ops.Fused8BitRowwiseQuantizedToFloat(x)
    if op == "dequantize4":
        return ops.FusedNBitRowwiseQuantizedSBHalfToFloat(x, 4)
    s["tables"].assign_rows_from_float(0, x)
    return s["tables"].weights_dev


# ---- what a pass cannot do without ----------------------------------------------------------------------

def _distinct(dist, rows, n):
    """Rows of a table that n looked-up rows are expected to touch: each has to be read once, however often it is named."""
    if dist == "uniform":
        return rows * -math.expm1(n * math.log1p(-1.0 / rows)) if rows > 1 else 1.0
    edges = torch.arange(1, rows + 2, dtype=torch.float64).pow_(1.0 - float(dist.split(":")[1]))
    p = (edges[:-1] - edges[1:]) / (edges[0] - edges[-1])
    return float(-torch.expm1(n * torch.log1p(-p.clamp_(max=1 - 1e-12))).sum())


def work(case):
    kind = case["kind"]
    if kind in ("lookup", "request"):
        ws = _spec(case, 0)
        per_table = ws.B * _mean_length(case["lengths"])
        n, total_d, isz = ws.T * per_table, sum(ws.dims), case["bits"] // 8
        read = per_table * (1 - case.get("pruned", 0.0))
        distinct = _distinct(case["indices"], ws.E, read)
        table_bytes = sum(distinct * row_bytes(ty, d, 1) for ty, d in zip(ws.tys, ws.dims))
        out = (n * max(ws.dims) if case["pooling"] == "none" else ws.B * total_d) * SIZES[case["output"]]
        # the request: indices and offsets (or, as it arrives, lengths), per-sample weights
        request = n * isz + (ws.T * ws.B + 1) * isz + (4 * n if ws.weighted else 0)
        return {"bytes": table_bytes + request + out, "flops": 2.0 * read * total_d}
    if kind == "input":
        bags, isz = case["tables"] * case["batch"], case["bits"] // 8
        n = bags * _mean_length(case["lengths"])
        return {"bytes": 2 * n * (isz + (4 if case["weighted"] else 0)) + 3 * bags * isz, "flops": bags}
    if kind == "order":
        dims = [int(d) for d in case["dims"].split(",")]
        n = case["batch"] * sum(dims[t % len(dims)] for t in range(case["tables"]))
        return {"bytes": 2 * n * SIZES[case["dtype"]] * (2 if case["backward"] else 1), "flops": 0}
    rows, cols, op = case["rows"], case["cols"], case["op"]
    coded = {"8": cols + (4 if op == "table8" else 8), "4": cols // 2 + 4}[op[-1]]
    return {"bytes": rows * (4 * cols + coded), "flops": 4.0 * rows * cols}


def tolerance(case):
    """Bytes and copies are exact, and so is a single row's code * scale + bias.  Pooled sums: four times what the listed
    cases are off by from the same sums in 64 bits (fp32 6.1e-6, the weighted 8-bit rows; fp16 2.1e-4; bf16 1.7e-3)."""
    if case["kind"] in ("input", "order", "rowwise") or case["pooling"] == "none":
        return "exact"
    return {"fp32": {"rel": 2.5e-5}, "fp16": {"rel": 8e-4}, "bf16": {"rel": 7e-3}}[case["output"]]


# ---- the same in 64 bits ----------------------------------------------------------------------------------

def _decoded(rows, ty, dim):
    """Table rows (bytes) as float64 [n, dim]."""
    n = rows.shape[0]
    if ty in ("fp32", "fp16"):
        dtype, size = (torch.float32, 4) if ty == "fp32" else (torch.float16, 2)
        return rows[:, :size * dim].contiguous().view(dtype).view(n, dim).double()
    if ty == "fp8":
        b = torch.arange(256, device=rows.device)
        e, m, sign = (b >> 3) & 15, (b & 7).double(), 1.0 - 2.0 * (b >> 7).double()
        values = sign * torch.where(e > 0, (1.0 + m / 8.0) * torch.exp2((e - 7).double()), m / 8.0 * 2.0 ** -6)
        return values[rows[:, :dim].long()]
    header = rows[:, :4].contiguous().view(torch.float16).view(n, 2).double()
    bits = {"int8": 8, "int4": 4, "int2": 2}[ty]
    shifts = torch.arange(0, 8, bits, device=rows.device, dtype=torch.uint8)
    codes = ((rows[:, 4:4 + (dim * bits + 7) // 8].unsqueeze(-1) >> shifts) & (2 ** bits - 1)).flatten(1)[:, :dim]
    return codes.double() * header[:, :1] + header[:, 1:]


def _exact_lookup(case, s, indices, offsets):
    ws, types = _spec(case, 0), case["types"].split(",")
    pooled, column = case["pooling"] != "none", 0
    bounds = offsets[:: ws.B].tolist()
    out = torch.zeros(ws.B if pooled else indices.numel(), sum(ws.dims) if pooled else max(ws.dims), dtype=torch.float64, device=indices.device)
    for t, dim in enumerate(ws.dims):
        rows, mine = s["tables"].table_rows(t), offsets[t * ws.B:(t + 1) * ws.B + 1].long()
        for lo in range(bounds[t], bounds[t + 1], 1 << 20):
            hi = min(bounds[t + 1], lo + (1 << 20))
            i = indices[lo:hi].long()
            x = _decoded(rows[i.clamp(min=0)], types[t % len(types)], dim) * (i >= 0).unsqueeze(1)
            if not pooled:
                out[lo:hi, :dim] = x
                continue
            if s["weights"] is not None:
                x *= s["weights"][lo:hi].unsqueeze(1)
            bag = torch.searchsorted(mine, torch.arange(lo, hi, device=i.device), right=True) - 1
            out[:, column:column + dim].index_add_(0, bag, x)
        if case["pooling"] == "mean":
            out[:, column:column + dim] /= (mine[1:] - mine[:-1]).clamp(min=1).unsqueeze(1)
        column += dim
    return out


def exact(case, seed):
    """What ``run`` returns for these inputs, from the tables' bytes in float64; None where the outputs are bytes, indices
    or copies."""
    kind = case["kind"]
    if kind not in ("lookup", "request") and not (kind == "rowwise" and case["op"].startswith("dequantize")):
        return None
    s = prepare(case, seed)
    if kind == "lookup":
        return _exact_lookup(case, s, s["indices"], s["offsets"])
    if kind == "rowwise":
        x = s["x"]
        if case["op"] == "dequantize8":
            header = x[:, -8:].contiguous().view(torch.float32).double()
            return x[:, :-8].double() * header[:, :1] + header[:, 1:]
        return _decoded(torch.cat([x[:, -4:], x[:, :-4]], 1), "int4", case["cols"])
    order = s["permute"].tolist()
    parts = torch.split(s["values"], s["lengths"].sum(1).tolist())
    lengths = s["lengths"][s["permute"].long()].view(-1)
    offsets = torch.zeros(lengths.numel() + 1, dtype=torch.int64, device=lengths.device)
    offsets[1:] = torch.cumsum(lengths, 0)
    pooled = _exact_lookup(case, s, torch.cat([parts[t] for t in order]), offsets)
    pieces = torch.split(pooled, _spec(case, 0).dims, 1)
    return torch.cat([pieces[f] for f in s["order"]._permute.tolist()], 1)
