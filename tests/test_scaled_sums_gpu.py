"""Rows and weights at the ends of fp32's range.  The lookup keeps its sums scaled by a power of two, which is exact
while every weighted scale and bias is zero or of magnitude 2^-68 to 2^36; bags with other values take another path,
their neighbours in the same warp do not.  Bit for bit against the CPU oracle (NaN where the oracle has NaN)."""
import numpy as np
import pytest
import torch

import fbgemm_b200 as F
from conftest import bits
from helpers import random_fused_table

pytestmark = pytest.mark.gpu
BELOW = np.nextafter(np.float32(1), np.float32(0))
FLOATS = np.array([0.0, -0.0, 2.0**-52, 2.0**-52 * BELOW, -2.0**-52, 2.0**52, 2.0**52 * BELOW, -2.0**52, 2.0**-53, 1e-20, -1e-20, 1e20,
                   3e38, -3e38, 1e-44, 2.0**-126, 2.0**-75, 2.0**-74, 2.0**-149, np.inf, -np.inf, np.nan,
                   2.0**-68, 2.0**-68 * BELOW, -2.0**-68, 2.0**36, 2.0**36 * BELOW, -2.0**36, 2.0**-91, 2.0**-59], np.float32)
HALVES = np.array([0.0, -0.0, 2.0**-24, -2.0**-24, 2.0**-14, 65504.0, -65504.0, np.inf, -np.inf, np.nan], np.float16)


def dev(a):
    return None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()


def same(got, ref):
    np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
    fine = ~np.isnan(ref)
    np.testing.assert_array_equal(bits(got)[fine], bits(ref)[fine])


def make(rng, bit_rate, dim, batch, weighted, ordinary, sb_last=True):
    """Rows 0 .. 99 are ordinary; each of the others has an odd scale, bias or both, and every fourth bag names one.
    Rows 200 .. 239 cancel one another: payload 0 and biases b, -b (of sizes that meet in the sums' last places)."""
    rows = 240
    t = random_fused_table(rng, rows, dim, bit_rate, scale_bias_first=not sb_last)
    odd, kind = (FLOATS, np.float32) if bit_rate == 8 and sb_last else (HALVES, np.float16)
    width = 2 * kind().itemsize
    at, payload = (slice(-width, None), slice(0, -width)) if sb_last else (slice(0, width), slice(width, None))
    sb = np.ascontiguousarray(t[:, at]).view(kind)
    sb[100:200] = rng.choice(odd, (100, 2))
    sb[100:140, 0] = sb[:40, 0]
    sb[140:180, 1] = sb[:40, 1]
    t[200:, payload] = 0
    size = (2.0 ** rng.integers(-66 if kind == np.float32 else -14, 36 if kind == np.float32 else 15, 20)).astype(kind)
    sb[200::2, 1], sb[201::2, 1] = size, -size
    t[:, at] = sb.view(np.uint8)
    lengths = rng.integers(0, 40, batch)
    n = int(lengths.sum())
    indices = rng.choice(np.concatenate([np.arange(100), np.arange(200, rows)]), n)
    offsets = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    w = rng.standard_normal(n).astype(np.float32) if weighted else None
    if not ordinary:
        for b in range(0, batch, 4):
            if lengths[b]:
                indices[rng.integers(offsets[b], offsets[b + 1])] = rng.integers(100, 200)
        for b in range(2, batch, 4):
            if weighted and lengths[b]:
                w[rng.integers(offsets[b], offsets[b + 1])] = rng.choice(FLOATS)
    return rows, t, indices, offsets, w, n


@pytest.mark.parametrize("bit_rate", [8, 4, 2])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("ordinary", [False, True])
def test_one_table(gpu_ctx, oracle, bit_rate, weighted, ordinary):
    rng = np.random.default_rng(10 * bit_rate + 2 * weighted + ordinary)
    for dim in (4, 20, 64, 128, 256, 300):
        many = 15_000 if dim <= 128 else 3000
        for batch, mean in ((50, False), (50, True), (1500, False), (1500, True), (many, False), (many, True)):
            rows, t, indices, offsets, w, n = make(rng, bit_rate, dim, batch, weighted, ordinary)
            with np.errstate(all="ignore"):
                ok_ref, ref = oracle.spmdm(bit_rate, dim, rows, t, indices, offsets, w, mean, np.float32, False, True,
                                           output_size=batch, index_size=n)
            kw = dict(index_dtype=np.int64, offset_dtype=np.int32, out_dtype=np.float32)
            kern = (F.GenerateEmbeddingSpMDM(dim, weighted, mean, **kw) if bit_rate == 8
                    else F.GenerateEmbeddingSpMDMNBit(bit_rate, dim, weighted, mean, **kw))
            out = torch.zeros(batch * dim, device="cuda")
            assert kern(batch, n, rows, dev(t), dev(indices), dev(offsets), dev(w), out) and ok_ref
            same(out.cpu().numpy(), ref)


@pytest.mark.parametrize("bit_rate", [8, 4, 2])
@pytest.mark.parametrize("form", ["sb_first", "lengths", "positional"])
def test_other_forms(gpu_ctx, oracle, bit_rate, form):
    rng = np.random.default_rng(100 * bit_rate + len(form))
    sb_last, use_offsets, positional = form != "sb_first", form != "lengths", form == "positional"
    for dim in (20, 64, 128, 256):
        for batch, mean in ((1500, False), (1500, True), (15_000 if dim <= 128 else 3000, True)):
            weighted = positional or mean
            rows, t, indices, offsets, w, n = make(rng, bit_rate, dim, batch, weighted, False, sb_last)
            if not sb_last:
                indices[rng.random(n) < 0.2] = -1
            if positional:
                w = rng.standard_normal(40).astype(np.float32)
                w[rng.integers(0, 40, 3)] = rng.choice(FLOATS[FLOATS != 0], 3)
            ol = offsets if use_offsets else np.diff(offsets).astype(np.int32)
            with np.errstate(all="ignore"):
                ok_ref, ref = oracle.spmdm_ex(bit_rate, dim, rows, t, indices, ol, w, mean, "f32", positional, use_offsets, -1, -1,
                                              sb_last, False, output_size=batch, index_size=n)
            kw = dict(index_dtype=np.int64, offset_dtype=np.int32)
            args = (dim, weighted, mean, 16, positional, use_offsets, -1, -1, sb_last)
            kern = (F.GenerateEmbeddingSpMDMWithStrides(*args, **kw) if bit_rate == 8
                    else F.GenerateEmbeddingSpMDMNBitWithStrides(bit_rate, *args, **kw))
            out = torch.zeros(batch * dim, device="cuda")
            assert kern(batch, n, rows, dev(t), dev(indices), dev(ol), dev(w), out) and ok_ref
            same(out.cpu().numpy(), ref[:batch * dim])


@pytest.mark.parametrize("bit_rate", [8, 4, 2])
@pytest.mark.parametrize("batch", [1500, 15_000])
def test_rows_beyond_4gb(gpu_ctx, oracle, bit_rate, batch):
    """Odd rows on both sides of 4 GB: behind a pruning map, which names them beside ordinary and pruned ones, and in a table
    of 64-bit row offsets, alone and beside a small table in one launch."""
    rng = np.random.default_rng(bit_rate + batch)
    dim, stride, total = 128, 40_960, 120_000
    rows, t, indices, offsets, w, n = make(rng, bit_rate, dim, batch, True, False)
    used = np.sort(rng.choice(total, rows, replace=False))
    used[-1] = total - 1
    big = torch.zeros(total * stride, dtype=torch.uint8, device="cuda").view(total, stride)
    big[torch.from_numpy(used).cuda(), :t.shape[1]] = dev(t)
    kw = dict(index_dtype=np.int64, offset_dtype=np.int32)
    for mean in (False, True):
        # a map of rows and pruned ones; the functor's rows lie one behind the other, so the map names parts of the pitch
        parts = t.shape[1]
        per_row = stride // parts
        flat = torch.zeros((total * per_row, parts), dtype=torch.uint8, device="cuda")
        at = used * per_row
        flat[torch.from_numpy(at).cuda()] = dev(t)
        cit = np.concatenate([np.arange(rows), np.full(60, -1)]).astype(np.int32)
        idx = indices.copy()
        gone = rng.random(n) < 0.2
        idx[gone] = rng.integers(rows, rows + 60, int(gone.sum()))
        with np.errstate(all="ignore"):
            ok_ref, ref = oracle.spmdm_rowwise_sparse(bit_rate, dim, rows + 60, t, idx, cit, offsets, w, mean)
        kern = (F.GenerateEmbeddingSpMDMRowWiseSparse(dim, True, mean, **kw) if bit_rate == 8
                else F.GenerateEmbeddingSpMDMNBitRowWiseSparse(bit_rate, dim, True, mean, **kw))
        far = np.where(cit >= 0, at[np.minimum(cit, rows - 1)], -1).astype(np.int32)
        out = torch.zeros(batch * dim, device="cuda")
        assert kern(batch, n, rows + 60, flat, dev(idx), dev(offsets), dev(w), out, dev(far)) and ok_ref
        same(out.cpu().numpy(), ref[:batch * dim])
        del flat

        with np.errstate(all="ignore"):
            ok_ref, ref = oracle.spmdm(bit_rate, dim, rows, t, indices, offsets, w, mean, np.float32, False, True,
                                       output_size=batch, index_size=n)
        args = (dim, True, mean, 16, False, True, -1)
        gen = (F.GenerateEmbeddingSpMDMWithStrides if bit_rate == 8
               else lambda *a, **k: F.GenerateEmbeddingSpMDMNBitWithStrides(bit_rate, *a, **k))
        wide, narrow = gen(*args, stride, True, **kw), gen(*args, -1, True, **kw)
        out = torch.zeros(batch * dim, device="cuda")
        assert wide(batch, n, total, big, dev(used[indices]), dev(offsets), dev(w), out) and ok_ref
        same(out.cpu().numpy(), ref)
        outs = [torch.zeros_like(out) for _ in range(2)]
        plan = F.MultiTablePlan([(wide, batch, n, total, big, dev(used[indices]), dev(offsets), dev(w), outs[0], None),
                                 (narrow, batch, n, rows, dev(t), dev(indices), dev(offsets), dev(w), outs[1], None)])
        plan.launch()
        assert F.status_read(0)[0]
        for o in outs:
            same(o.cpu().numpy(), ref)
        plan.close()


@pytest.mark.parametrize("weighted", [False, True])
def test_several_tables(gpu_ctx, oracle, weighted):
    rng = np.random.default_rng(3 + weighted)
    calls, want = [], []
    for t in range(9):
        bit_rate, dim, batch = (8, 4, 2)[t % 3], (64, 128, 256)[t // 3], 70 + t
        rows, table, indices, offsets, w, n = make(rng, bit_rate, dim, batch, weighted, t == 4)
        want.append(oracle.spmdm(bit_rate, dim, rows, table, indices, offsets, w, False, np.float32, False, True,
                                 output_size=batch, index_size=n)[1])
        kw = dict(index_dtype=np.int64, offset_dtype=np.int32, out_dtype=np.float32)
        kern = (F.GenerateEmbeddingSpMDM(dim, weighted, False, **kw) if bit_rate == 8
                else F.GenerateEmbeddingSpMDMNBit(bit_rate, dim, weighted, False, **kw))
        calls.append((kern, batch, n, rows, dev(table), dev(indices), dev(offsets), dev(w), torch.zeros(batch * dim, device="cuda"), None))
    plan = F.MultiTablePlan(calls)
    plan.launch()
    assert F.status_read(0)[0]
    for c, ref in zip(calls, want):
        same(c[8].cpu().numpy(), ref)
    plan.close()


@pytest.mark.parametrize("bit_rate,dim,batch", [(8, 128, 10_000), (4, 64, 4096)])
def test_small_weights_cost_nothing(gpu_ctx, bit_rate, dim, batch):
    """Per-sample weights of 1e-16, which decay and softmax produce, are as fast as others.  (When only magnitudes from
    2^-52 on entered the scaled sums, such bags were pooled twice: 1.8 and 2.8 times the time.  Half as long again leaves
    room for a clock that changes between the two.)"""
    rng = np.random.default_rng(bit_rate)
    rows, length = 100_000, 20
    n = batch * length
    table = random_fused_table(rng, rows, dim, bit_rate)
    kind = np.float32 if bit_rate == 8 else np.float16
    table[:, -2 * kind().itemsize:] = rng.uniform(0.5, 1.5, (rows, 2)).astype(kind).view(np.uint8)
    table = dev(table)
    indices, offsets = dev(rng.integers(0, rows, n)), dev(np.arange(0, n + 1, length).astype(np.int32))
    out = torch.zeros(batch * dim, device="cuda")
    kw = dict(index_dtype=np.int64, offset_dtype=np.int32, out_dtype=np.float32)
    kern = F.GenerateEmbeddingSpMDM(dim, True, False, **kw) if bit_rate == 8 else F.GenerateEmbeddingSpMDMNBit(bit_rate, dim, True, False, **kw)

    def best_of(weights, begin=torch.cuda.Event(enable_timing=True), end=torch.cuda.Event(enable_timing=True)):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            kern.launch(batch, n, rows, table, indices, offsets, weights, out)
        torch.cuda.synchronize()
        graph, times = torch.cuda.CUDAGraph(), []
        with torch.cuda.graph(graph, stream=stream):
            for _ in range(50):
                kern.launch(batch, n, rows, table, indices, offsets, weights, out)
        for _ in range(5):
            begin.record()
            graph.replay()
            end.record()
            torch.cuda.synchronize()
            times.append(begin.elapsed_time(end))
        return min(times)

    w = (0.5 + torch.rand(n, device="cuda"))
    usual, small = best_of(w), best_of(w * 1e-16)
    assert small < 1.5 * usual, (small, usual)
