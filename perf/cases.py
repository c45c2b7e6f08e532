"""What this package is used for, as cases that can be timed: pooled lookups in
one table (called and awaited, or enqueued), in many tables at once (device and
host arrays, both row layouts), row-wise lookups without pooling, pruned tables,
and the quantizers that build the rows.

``listed()`` holds one case for each use, ``draw(rng)`` gives further ones over
the same ranges.  ``prepare`` builds the tables, the kernels and one set of
index arrays from a seed; ``run`` is one pass through the public entry points.

Tables are random rows with scales and biases as quantized N(0,1) rows have
them.  Indices are uniform or Zipf-distributed over scattered rows, bag lengths
fixed, uniform or Poisson - the distributions of ``fbgemm_b200.workloads`` and
of the lookup tests.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import fbgemm_b200 as F
from fbgemm_b200 import tbe
from fbgemm_b200 import workloads as W

ST = tbe.SparseType
TORCH = {"int32": torch.int32, "int64": torch.int64, "float32": torch.float32, "float16": torch.float16,
         "bfloat16": torch.bfloat16}
ESIZE = {"int32": 4, "int64": 8, "float32": 4, "float16": 2, "bfloat16": 2}
#: Row formats of the tables of a table-batched call, table t taking entry t modulo the length.
MIXES = {
    "int4": (ST.INT4,),
    "int8": (ST.INT8,),
    "mixed": (ST.INT8, ST.INT4, ST.INT2),                                        # the quantized formats alone
    "serving": (ST.INT8, ST.INT4, ST.INT4, ST.FP16, ST.INT8, ST.INT2, ST.INT4, ST.FP8),  # with unquantized tables among them
}
DIMS = {"64_128_256": (64, 128, 256), "128": (128,), "odd": (36, 100, 52, 164)}


# ---- the cases ---------------------------------------------------------------

def listed():
    return [
        # The generated kernel called as the CPU library is called, a handful of bags at a time, and its answer
        # awaited: the shape of the reference library's lookup benchmark (batch 10, about 100 rows a bag).
        dict(name="functor_8bit_d64_b10", use="functor", bits=8, dim=64, rows=4_000_000, batch=10, mean_len=100,
             lengths="uniform", alpha=0.0, weighted=False, mean=False, index="int64", offset="int32", out="float32",
             use_offsets=True),
        # One ranking-model table, 8-bit, fixed pooling, uniform indices; enqueued without waiting.
        dict(name="lookup_8bit_1Mx128_b10000", use="lookup", bits=8, dim=128, rows=1_000_000, batch=10_000, mean_len=20,
             lengths="fixed", alpha=0.0, weighted=False, mean=False, index="int64", offset="int64", out="float32",
             use_offsets=True),
        # One large 4-bit table, ragged bags with empty ones among them, per-sample weights, half output.
        dict(name="lookup_4bit_10Mx64_b4096", use="lookup", bits=4, dim=64, rows=10_000_000, batch=4_096, mean_len=32,
             lengths="ragged", alpha=1.05, weighted=True, mean=False, index="int32", offset="int32", out="float16",
             use_offsets=True),
        # Row width and batch that fit no tile, lengths instead of offsets, positions averaged, bfloat16 output.
        dict(name="lookup_8bit_300Kx86_lengths", use="lookup", bits=8, dim=86, rows=300_007, batch=3_001, mean_len=25,
             lengths="poisson", alpha=1.05, weighted=True, mean=True, index="int64", offset="int32", out="bfloat16",
             use_offsets=False),
        # A pruned 2-bit table: half of the logical rows are gone, indices go through the row map, mean pooling.
        dict(name="pruned_2bit_20Mx128_b8192", use="pruned", bits=2, dim=128, rows=20_000_000, batch=8_192, mean_len=30,
             lengths="poisson", alpha=1.1, weighted=False, mean=True, index="int64", offset="int64", out="float32",
             keep=0.5),
        # Serving one request batch: many tables of several row formats, few bags each.
        dict(name="tbe_serving_64x512", use="tbe", tables=64, rows=200_000, batch=512, mean_len=20, mix="serving",
             dims="64_128_256", weighted=False, mean=False, index="int32", out="float16", sb_last=False, align=16,
             alpha=1.05, pruned=False),
        # A trained model's table set at full batch, fused rows, one ordered step on device arrays.
        dict(name="tables_mixed_64x16384", use="tables", tables=64, rows=4_500_000, batch=16_384, mean_len=30,
             lengths="poisson", mix="mixed", dims="64_128_256", weighted=False, index="int32", out="float16", alpha=1.05),
        # The largest: a share of a 4-bit table set of 40 M rows each, global batch, weighted, fixed pooling.
        dict(name="tbe_int4_8x40M_b65536", use="tbe", tables=8, rows=40_000_000, batch=65_536, mean_len=40, mix="int4",
             dims="128", weighted=True, mean=False, index="int64", out="float16", sb_last=True, align=1, alpha=1.1,
             pruned=False),
        # Rows without pooling, for sequence models: one output row per index.
        dict(name="sequence_int8_8x32768", use="sequence", tables=8, rows=2_000_000, batch=32_768, mean_len=16, mix="int8",
             dim=128, index="int32", out="float16", sb_last=False, align=16, alpha=1.05),
        # Pruned table-batched tables: sparse to dense index through hash maps, then the pooled lookup, in which
        # the pruned indices (-1) are skipped.
        dict(name="hashed_tbe_16x4096", use="hashed", tables=16, rows=2_000_000, batch=4_096, mean_len=30, mix="int4",
             dims="128", weighted=False, mean=False, index="int64", out="float16", sb_last=False, align=16, alpha=1.05,
             map="hash", keep=0.5),
        # Building a table: fp32 rows to fused 8-bit rows.
        dict(name="quantize_8bit_1Mx128", use="quantize", bits=8, dim=128, rows=1_000_000),
        # The generated kernel on host arrays, as a program written for the CPU library calls it.
        dict(name="host_8bit_1Mx128_b10000", use="host", bits=8, dim=128, rows=1_000_000, batch=10_000, mean_len=20,
             lengths="fixed", alpha=0.0, weighted=False, mean=False, index="int64", offset="int64", out="float32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of a use that listed() stands for."""
    use = rng.choice(["functor", "lookup", "lookup", "odd", "pruned", "tbe", "tbe", "tables", "sequence", "hashed",
                      "quantize", "host"])
    ints = rng.choice(["int32", "int64"])
    coin = lambda: rng.random() < 0.5  # noqa: E731
    if use == "functor":
        return dict(use=use, bits=rng.choice([8, 4, 2]), dim=rng.choice([32, 40, 48, 64, 86, 128, 164, 256, 512, 1024]),
                    rows=_log(rng, 4_000, 4_000_000), batch=_log(rng, 1, 100), mean_len=_log(rng, 4, 100),
                    lengths="uniform", alpha=0.0, weighted=coin(), mean=coin(), index=ints, offset=rng.choice(["int32", "int64"]),
                    out=rng.choice(["float32", "float16"]), use_offsets=coin())
    if use in ("lookup", "odd"):
        dim = rng.choice([32, 48, 64, 96, 128, 256, 512]) if use == "lookup" else rng.randint(5, 300)
        return dict(use="lookup", bits=rng.choice([8, 4, 2]), dim=dim, rows=_log(rng, 40_000, 10_000_000),
                    batch=_log(rng, 300, 20_000), mean_len=rng.randint(5, 60),
                    lengths=rng.choice(["fixed", "ragged", "poisson"]), alpha=rng.choice([0.0, 1.05, 1.1]), weighted=coin(),
                    mean=coin(), index=ints, offset=rng.choice(["int32", "int64"]),
                    out=rng.choice(["float32", "float16", "bfloat16"]), use_offsets=coin())
    if use == "pruned":
        return dict(use=use, bits=rng.choice([8, 4, 2]), dim=rng.choice([64, 100, 128, 256]),
                    rows=_log(rng, 200_000, 20_000_000), batch=_log(rng, 300, 20_000), mean_len=rng.randint(5, 60),
                    lengths=rng.choice(["fixed", "ragged", "poisson"]), alpha=rng.choice([1.05, 1.1]), weighted=coin(),
                    mean=coin(), index=ints, offset=rng.choice(["int32", "int64"]), out="float32",
                    keep=rng.choice([0.3, 0.5, 0.8]))
    if use == "tbe":
        tables, batch = _log(rng, 4, 128), _log(rng, 64, 16_384)
        while tables * batch > 1 << 19:
            batch //= 2
        return dict(use=use, tables=tables, rows=min(_log(rng, 20_000, 2_000_000), 40_000_000 // tables), batch=batch, mean_len=rng.randint(5, 40),
                    mix=rng.choice(["serving", "mixed", "int4", "int8"]), dims=rng.choice(["64_128_256", "128", "odd"]),
                    weighted=coin(), mean=coin(), index=ints, out=rng.choice(["float16", "float16", "float32", "bfloat16"]),
                    sb_last=coin(), align=rng.choice([4, 16]), alpha=1.05, pruned=coin())
    if use == "tables":
        return dict(use=use, tables=_log(rng, 4, 64), rows=_log(rng, 100_000, 4_000_000), batch=_log(rng, 512, 16_384),
                    mean_len=rng.randint(5, 30), lengths=rng.choice(["fixed", "ragged", "poisson"]),
                    mix=rng.choice(["mixed", "int4", "int8"]), dims=rng.choice(["64_128_256", "128", "odd"]), weighted=coin(),
                    index=ints, out=rng.choice(["float16", "float32"]), alpha=rng.choice([1.05, 1.1]))
    if use == "sequence":
        tables, batch, mean_len = _log(rng, 1, 16), _log(rng, 256, 32_768), rng.randint(4, 30)
        dim, out = rng.choice([32, 64, 100, 128, 256]), rng.choice(["float16", "float32", "bfloat16"])
        while tables * batch * mean_len * dim * ESIZE[out] > 1 << 30:
            batch //= 2
        return dict(use=use, tables=tables, rows=_log(rng, 20_000, 2_000_000), batch=batch, mean_len=mean_len,
                    mix=rng.choice(["int8", "int4", "serving"]), dim=dim, index=ints, out=out, sb_last=coin(),
                    align=rng.choice([4, 16]), alpha=1.05)
    if use == "hashed":
        return dict(use=use, tables=_log(rng, 2, 16), rows=_log(rng, 50_000, 2_000_000), batch=_log(rng, 256, 8_192),
                    mean_len=rng.randint(5, 40), mix=rng.choice(["int4", "int8", "mixed"]), dims=rng.choice(["128", "64_128_256"]),
                    weighted=coin(), mean=coin(), index=ints, out=rng.choice(["float16", "float32"]), sb_last=False, align=16,
                    alpha=1.05, map=rng.choice(["hash", "array"]), keep=rng.choice([0.3, 0.5, 0.8]))
    if use == "quantize":
        bits = rng.choice([8, 4, 2])
        dim = rng.choice([64, 128, 256, rng.randint(5, 400)])
        return dict(use=use, bits=bits, dim=(dim + 8 // bits - 1) // (8 // bits) * (8 // bits), rows=_log(rng, 1_000, 1_500_000))
    return dict(use="host", bits=rng.choice([8, 4, 2]), dim=rng.choice([64, 86, 128]), rows=_log(rng, 20_000, 1_000_000),
                batch=_log(rng, 100, 20_000), mean_len=rng.randint(5, 40), lengths=rng.choice(["fixed", "ragged", "poisson"]),
                alpha=rng.choice([0.0, 1.05]), weighted=coin(), mean=coin(), index=ints, offset=rng.choice(["int32", "int64"]),
                out=rng.choice(["float32", "float16"]))


# ---- inputs --------------------------------------------------------------------

def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _gen(seed, device):
    return torch.Generator(device=device).manual_seed(int(seed) & 0x7FFFFFFF)


def _random_bytes(n, g, dev):
    words = torch.randint(-(1 << 63), (1 << 63) - 1, ((n + 7) // 8,), generator=g, device=dev, dtype=torch.int64)
    return words.view(torch.uint8)[:n]


#: scale of a quantized N(0,1) row (its range over the number of steps), bias about the row's minimum
SCALE = {8: 0.02, 4: 0.33, 2: 1.6}


def _write_scale_bias(rows2d, at, bits, half, g):
    """Scale and bias of every row of ``rows2d`` ([rows, row bytes] uint8) at byte ``at``."""
    n = rows2d.shape[0]
    sb = torch.rand((n, 2), generator=g, device=rows2d.device)
    sb[:, 0] = (0.7 + 0.6 * sb[:, 0]) * SCALE[bits]
    sb[:, 1] = -2.0 - sb[:, 1]
    sb = sb.half() if half else sb
    width = 4 if half else 8
    rows2d[:, at:at + width] = sb.view(torch.uint8).view(n, width)


def _fused_table(rows, dim, bits, g, dev):
    row_bytes = W.fused_row_bytes(bits, dim)
    t = _random_bytes(rows * row_bytes, g, dev).view(rows, row_bytes)
    _write_scale_bias(t, row_bytes - (8 if bits == 8 else 4), bits, bits != 8, g)
    return t


def _lengths(kind, mean_len, n, g, dev):
    if kind == "fixed":
        return torch.full((n,), int(mean_len), device=dev, dtype=torch.int64)
    if kind == "ragged":    # empty bags among them
        return torch.randint(0, 2 * mean_len + 1, (n,), generator=g, device=dev, dtype=torch.int64)
    if kind == "uniform":
        return torch.randint(1, 2 * mean_len, (n,), generator=g, device=dev, dtype=torch.int64)
    return torch.poisson(torch.full((n,), float(mean_len), device=dev), generator=g).to(torch.int64)


def _indices(n, rows, alpha, seed, g, dev):
    """n row numbers below ``rows`` (a number, or a tensor of n numbers): uniform, or Zipf ranks scattered over the
    rows by a multiplication with a prime above every row count."""
    if alpha <= 1.0:
        u = torch.rand(n, generator=g, device=dev, dtype=torch.float64)
        return (u * rows).to(torch.int64)
    z = (W.zipf(n, alpha, dev, int(seed) & 0x7FFFFFFF) - 1) % rows
    return z * 2654435761 % rows


def _mix(case):
    tys = MIXES[case["mix"]]
    dims = DIMS[case["dims"]] if "dims" in case else (case["dim"],)
    T = case["tables"]
    # widths change once the row formats have gone round, so that every format meets every width
    return [tys[t % len(tys)] for t in range(T)], [dims[(t // len(tys)) % len(dims)] for t in range(T)]


def _table_rows(case):
    """Row counts of the tables: a third, the nominal count and 5/3 of it in turn."""
    return [max(16, case["rows"] * (1 + 2 * (t % 3)) // 3) if case["tables"] > 8 else case["rows"]
            for t in range(case["tables"])]


def _row_bytes(case, ty, dim):
    sb = 8 if (ty == ST.INT8 and case.get("sb_last", True)) else 4
    return tbe.padded_row_size_in_bytes(dim, ty, case.get("align", 1), sb)


def _blob(case, tys, dims, rows, g, dev):
    """The tables of a table-batched operator in one block of bytes, and where each starts."""
    rb = [_row_bytes(case, ty, d) for ty, d in zip(tys, dims)]
    starts = np.concatenate([[0], np.cumsum([r * b for r, b in zip(rows, rb)])]).astype(np.int64)
    blob = _random_bytes(int(starts[-1]), g, dev)
    for t, (ty, d) in enumerate(zip(tys, dims)):
        view = blob[int(starts[t]):int(starts[t + 1])].view(rows[t], rb[t])
        if ty in tbe._BITS:
            bits = tbe._BITS[ty]
            half = not (ty == ST.INT8 and case["sb_last"])
            _write_scale_bias(view, d * bits // 8 if case["sb_last"] else 0, bits, half, g)
        elif ty == ST.FP8:
            view &= 0xBF    # exponents of magnitudes below 2
        elif ty == ST.FP16:
            view[:, :2 * d] = torch.randn((rows[t], d), generator=g, device=dev).half().view(torch.uint8).view(rows[t], 2 * d)
    return blob, starts[:-1]


def _batched_indices(case, rows, kind, seed, g, dev):
    """(indices, offsets[T*B+1], positions of each table) of a table-batched call."""
    T, B = case["tables"], case["batch"]
    lengths = _lengths(kind, case["mean_len"], T * B, g, dev)
    n = T * B * case["mean_len"]
    while (short := n - int(lengths.sum())) != 0:   # the same number of positions, hence output rows, for every seed
        bags = torch.arange(T * B, device=dev) if short > 0 else lengths.nonzero()[:, 0]
        bags = bags[torch.randperm(bags.numel(), generator=g, device=dev)[:abs(short)]]
        lengths[bags] += 1 if short > 0 else -1
    offsets = W.offsets_from_lengths(lengths, torch.int64)
    counts = lengths.view(T, B).sum(1)
    per_pos = torch.repeat_interleave(torch.tensor(rows, device=dev, dtype=torch.int64), counts, output_size=n)
    indices = _indices(n, per_pos, case["alpha"], seed, g, dev)
    return indices, offsets, counts


# ---- prepare -------------------------------------------------------------------

def _single_arrays(case, rows, seed, g, dev):
    lengths = _lengths(case["lengths"], case["mean_len"], case["batch"], g, dev)
    offsets = W.offsets_from_lengths(lengths, TORCH[case["offset"]])
    n = int(offsets[-1])
    indices = _indices(n, rows, case["alpha"], seed, g, dev).to(TORCH[case["index"]])
    weights = torch.rand(n, generator=g, device=dev) if case["weighted"] else None
    return lengths.to(TORCH[case["offset"]]), offsets, indices, weights, n


def _single_kernel(case):
    np_of = {"int32": np.int32, "int64": np.int64, "float32": np.float32, "float16": np.float16, "bfloat16": np.uint16}
    kw = dict(index_dtype=np_of[case["index"]], offset_dtype=np_of[case["offset"]])
    offs = case.get("use_offsets", True)
    if case["use"] == "pruned":
        if case["bits"] == 8:
            return F.GenerateEmbeddingSpMDMRowWiseSparse(case["dim"], case["weighted"], case["mean"], **kw)
        return F.GenerateEmbeddingSpMDMNBitRowWiseSparse(case["bits"], case["dim"], case["weighted"], case["mean"], **kw)
    kw["out_dtype"] = np_of[case["out"]]
    bf16 = case["out"] == "bfloat16"
    if case["bits"] == 8:
        return F.GenerateEmbeddingSpMDM(case["dim"], case["weighted"], case["mean"], use_offsets=offs, is_bf16_out=bf16, **kw)
    return F.GenerateEmbeddingSpMDMNBitWithStrides(case["bits"], case["dim"], case["weighted"], case["mean"],
                                                   use_offsets=offs, is_bf16_out=bf16, **kw)


def _prepare_single(case, seed, g, dev):
    rows, use = case["rows"], case["use"]
    cit, dense = None, rows
    if use == "pruned":
        keep = torch.rand(rows, generator=g, device=dev) < case["keep"]
        cit = torch.where(keep, torch.cumsum(keep, 0, dtype=torch.int32) - 1, torch.full((), -1, dtype=torch.int32, device=dev))
        dense = int(keep.sum())
    table = _fused_table(max(dense, 1), case["dim"], case["bits"], g, dev)
    lengths, offsets, indices, weights, n = _single_arrays(case, rows, seed, g, dev)
    out = torch.zeros((case["batch"], case["dim"]), dtype=TORCH[case["out"]], device=dev)
    kernel = _single_kernel(case)
    if use == "host":
        host = lambda x: None if x is None else x.cpu().numpy()  # noqa: E731
        table, offsets, indices, weights, out = host(table), host(offsets), host(indices), host(weights), host(out)
        F.get_context().register_table(table)   # resident in HBM, as a program that keeps its tables does once
        args = (case["batch"], n, rows, table, indices, offsets, weights, out)
    else:
        ol = offsets if case.get("use_offsets", True) else lengths
        args = (case["batch"], n, rows, table, indices, ol, weights, out) + ((cit,) if use == "pruned" else ())
    return {"use": use, "kernel": kernel, "args": args, "out": out}


def _prepare_tbe(case, seed, g, dev):
    tys, dims = _mix(case)
    rows = _table_rows(case)
    blob, starts = _blob(case, tys, dims, rows, g, dev)
    hashed = case["use"] == "hashed"
    # with a map the caller's indices name sparse rows, of which the kept ones have a dense row
    sparse = [int(r / case["keep"]) for r in rows] if hashed else rows
    indices, offsets, counts = _batched_indices(case, sparse, "poisson", seed, g, dev)
    idt = TORCH[case["index"]]
    if not hashed and case["pruned"] and not case["sb_last"]:     # indices of pruned rows arrive as -1
        indices[torch.rand(indices.numel(), generator=g, device=dev) < 0.2] = -1
    op = tbe.IntNBitTableBatchedEmbeddingBags(
        blob, starts, [int(t) for t in tys], np.concatenate([[0], np.cumsum(dims)]), sum(dims),
        tbe.PoolingMode.MEAN if case["mean"] else tbe.PoolingMode.SUM, case["align"],
        {"float32": ST.FP32, "float16": ST.FP16, "bfloat16": ST.BF16}[case["out"]], case["sb_last"], case["weighted"], idt)
    weights = torch.rand(indices.numel(), generator=g, device=dev) if case["weighted"] else None
    s = {"use": case["use"], "op": op, "indices": indices.to(idt), "offsets": offsets.to(idt), "weights": weights}
    if hashed:
        # a random choice of rows[t] of the sparse[t] row numbers of each table, in order
        picked = [torch.randperm(m, generator=g, device=dev)[:r].sort().values for r, m in zip(rows, sparse)]
        if case["map"] == "hash":
            slots = np.concatenate([[0], np.cumsum([int(r / 0.8) + 1 for r in rows])]).astype(np.int64)
            table = torch.full((int(slots[-1]), 2), -1, dtype=torch.int32, device=dev)
            keys_at = torch.from_numpy(np.concatenate([[0], np.cumsum(rows)]).astype(np.int64)).to(dev)
            at = torch.from_numpy(slots).to(dev)
            dense = torch.cat([torch.arange(r, device=dev) for r in rows])
            ok = tbe.pruned_hashmap_insert(torch.cat(picked).to(idt), dense.to(idt), keys_at.to(idt), table, at)
            assert ok, "the hash map is full"
        else:
            table = torch.full((sum(sparse),), -1, dtype=torch.int32, device=dev)
            first = np.concatenate([[0], np.cumsum(sparse)]).astype(np.int64)
            for t, k in enumerate(picked):
                table[int(first[t]) + k] = torch.arange(rows[t], dtype=torch.int32, device=dev)
            at = torch.from_numpy(first).to(dev)
        s["map"], s["map_at"], s["hash"] = table, at, case["map"] == "hash"
    return s


def _prepare_tables(case, seed, g, dev):
    tys, dims = _mix(case)
    rows, B = _table_rows(case), case["batch"]
    idt = TORCH[case["index"]]
    np_idx = np.int32 if case["index"] == "int32" else np.int64
    np_out = np.float32 if case["out"] == "float32" else np.float16
    total = sum(dims)
    out = torch.zeros((B, total), dtype=TORCH[case["out"]], device=dev)
    indices, offsets, counts = _batched_indices(case, rows, case["lengths"], seed, g, dev)
    at = np.concatenate([[0], np.cumsum(counts.cpu().numpy())])
    indices = indices.to(idt)
    weights = torch.rand(indices.numel(), generator=g, device=dev) if case["weighted"] else None
    tables, col, idx, off, wts = [], 0, [], [], []
    for t, (ty, d) in enumerate(zip(tys, dims)):
        bits = tbe._BITS[ty]
        if bits == 8:
            k = F.GenerateEmbeddingSpMDMWithStrides(d, case["weighted"], False, 16, False, True, total, -1,
                                                    index_dtype=np_idx, offset_dtype=np_idx, out_dtype=np_out)
        else:
            k = F.GenerateEmbeddingSpMDMNBitWithStrides(bits, d, case["weighted"], False, 16, False, True, total, -1,
                                                        index_dtype=np_idx, offset_dtype=np_idx, out_dtype=np_out)
        tables.append((k, B, rows[t], _fused_table(rows[t], d, bits, g, dev),
                       out.data_ptr() + col * out.element_size(), 0))
        lo, hi = int(at[t]), int(at[t + 1])
        idx.append(indices[lo:hi])
        off.append((offsets[t * B:(t + 1) * B + 1] - lo).to(idt))
        wts.append(weights[lo:hi] if case["weighted"] else None)
        col += d
    call = F.MultiTableHostCall(tables, out, dev.index, 3)
    return {"use": "tables", "call": call, "arrays": call.device_args(idx, off, wts if case["weighted"] else None),
            "keep": (tables, idx, off, wts), "out": out}


def _prepare_sequence(case, seed, g, dev):
    tys, dims = _mix(case)
    rows = _table_rows(case)
    blob, starts = _blob(case, tys, dims, rows, g, dev)
    indices, offsets, _ = _batched_indices(case, rows, "poisson", seed, g, dev)
    op = tbe.IntNBitSequenceEmbedding(blob, starts, [int(t) for t in tys], case["dim"], case["align"],
                                      {"float32": ST.FP32, "float16": ST.FP16, "bfloat16": ST.BF16}[case["out"]],
                                      case["sb_last"])
    idt = TORCH[case["index"]]
    return {"use": "sequence", "op": op, "indices": indices.to(idt), "offsets": offsets.to(idt)}


def prepare(case, seed):
    dev = _dev()
    g = _gen(seed, dev)
    use = case["use"]
    if use in ("functor", "lookup", "pruned", "host"):
        return _prepare_single(case, seed, g, dev)
    if use in ("tbe", "hashed"):
        return _prepare_tbe(case, seed, g, dev)
    if use == "tables":
        return _prepare_tables(case, seed, g, dev)
    if use == "sequence":
        return _prepare_sequence(case, seed, g, dev)
    return {"use": "quantize", "bits": case["bits"],
            "x": torch.randn((case["rows"], case["dim"]), generator=g, device=dev)}


# ---- one pass ------------------------------------------------------------------

def run(state):
    use = state["use"]
    if use in ("functor", "host"):     # called and awaited: the bool is the call's answer
        ok = state["kernel"](*state["args"])
        return {"out": state["out"], "ok": ok}
    if use in ("lookup", "pruned"):
        state["kernel"].launch(*state["args"])
        return state["out"]
    if use == "tbe":
        return state["op"].forward(state["indices"], state["offsets"], state["weights"])
    if use == "hashed":
        lookup = tbe.pruned_hashmap_lookup if state["hash"] else tbe.pruned_array_lookup
        dense = lookup(state["indices"], state["offsets"], state["map"], state["map_at"])
        return {"dense": dense, "out": state["op"].forward(dense, state["offsets"], state["weights"])}
    if use == "tables":
        state["call"].step_device(state["arrays"], True, torch.cuda.current_stream().cuda_stream)
        return state["out"]
    if use == "sequence":
        return state["op"].forward(state["indices"], state["offsets"])
    if state["bits"] == 8:
        return F.FloatToFused8BitRowwiseQuantizedSBFloat(state["x"])
    return F.FloatToFusedNBitRowwiseQuantizedSBHalf(state["bits"], state["x"])


# ---- what a pass cannot do without ----------------------------------------------

def work(case):
    """Bytes: the rows an index names (each gathered row once), the indices, offsets, weights and map entries, and the
    output.  Operations: an addition and a multiply-add per pooled row and column."""
    use = case["use"]
    if use == "quantize":
        n = case["rows"] * case["dim"]
        return {"bytes": n * 4 + case["rows"] * W.fused_row_bytes(case["bits"], case["dim"]), "flops": 4 * n}
    if use in ("functor", "lookup", "pruned", "host"):
        n = case["batch"] * case["mean_len"]
        kept = n * case.get("keep", 1.0)
        b = kept * W.fused_row_bytes(case["bits"], case["dim"]) + n * ESIZE[case["index"]]
        b += case["batch"] * (ESIZE[case["offset"]] + case["dim"] * ESIZE[case["out"]])
        b += n * 4 if case["weighted"] else 0
        b += n * 4 if use == "pruned" else 0
        return {"bytes": b, "flops": 3 * kept * case["dim"]}
    tys, dims = _mix(case)
    n = case["batch"] * case["mean_len"]        # positions of one table
    idx, out = ESIZE[case["index"]], ESIZE[case["out"]]
    b = flops = 0.0
    for ty, d in zip(tys, dims):
        kept = n * (case["keep"] if use == "hashed" else 0.8 if case.get("pruned") and not case["sb_last"] else 1.0)
        unpadded = (d * tbe._BITS[ty] / 8 + (8 if ty == ST.INT8 and case.get("sb_last", True) else 4)) if ty in tbe._BITS \
            else d * tbe._PLAIN_BYTES[ty]
        b += kept * unpadded + n * idx + case["batch"] * idx
        if use == "sequence":
            b += n * d * out
            flops += 2 * n * d
            continue
        b += case["batch"] * d * out + (n * 4 if case["weighted"] else 0)
        flops += 3 * kept * d
        if use == "hashed":     # the map's entry (key and value, or value), and the dense index that is returned
            b += n * ((8 if case["map"] == "hash" else 4) + idx)
    return {"bytes": b, "flops": flops}


def tolerance(case):
    """Rounding of the output type; sums of 32-bit values are good to about 1e-5.  Quantized rows are bytes."""
    if case["use"] == "quantize":
        return "exact"
    return {"rel": {"float32": 1e-5, "float16": 5e-4, "bfloat16": 4e-3}[case["out"]]}
