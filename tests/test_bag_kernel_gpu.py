"""The pooled lookup at the edges of its kernels: row widths around the column
tiles, every alignment of a row, bags around the 32 (16, 8) indices a lane group
walks at a time, batches for whole, half and quarter warps per bag, rows beyond
4 GB, and more tables than one launch takes.  Bit for bit against the CPU
oracle."""
import numpy as np
import pytest
import torch

import fbgemm_b200 as F
from conftest import bits
from helpers import random_fused_table, row_bytes

pytestmark = pytest.mark.gpu
EDGE_LENGTHS = np.array([0, 1, 3, 4, 5, 7, 8, 9, 12, 15, 16, 17, 31, 32, 33, 47, 64, 65])


def dev(a):
    return None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()


def generate(bit_rate, dim, weighted, sb_last, stride):
    kw = dict(index_dtype=np.int64, offset_dtype=np.int32, out_dtype=np.float32)
    if bit_rate == 8:
        return F.GenerateEmbeddingSpMDMWithStrides(dim, weighted, False, 16, False, True, -1, stride, sb_last, **kw)
    return F.GenerateEmbeddingSpMDMNBitWithStrides(bit_rate, dim, weighted, False, 16, False, True, -1, stride, sb_last, **kw)


def check(oracle, rng, bit_rate, dim, batch, sb_last, pad, weighted=True, rows=150):
    natural = (dim * bit_rate + 7) // 8 + (8 if bit_rate == 8 and sb_last else 4)
    stride = natural + pad
    table = random_fused_table(rng, rows, dim, bit_rate, stride, not sb_last)
    lengths = rng.choice(EDGE_LENGTHS, batch) if batch < 1000 else rng.integers(0, 4, batch)
    if batch >= 1000:
        lengths[rng.integers(0, batch, 60)] = rng.choice(EDGE_LENGTHS, 60)
    n = int(lengths.sum())
    indices = rng.integers(0, rows, n)
    if not sb_last:
        indices[rng.random(n) < 0.3] = -1
    offsets = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    w = rng.standard_normal(n).astype(np.float32) if weighted else None
    ok_ref, ref = oracle.spmdm_ex(bit_rate, dim, rows, table, indices, offsets, w, False, "f32", False, True, -1, stride,
                                  sb_last, False, output_size=batch, index_size=n)
    out = torch.ones(batch * dim + 8, device="cuda")
    ok = generate(bit_rate, dim, weighted, sb_last, stride)(batch, n, rows, dev(table), dev(indices), dev(offsets), dev(w), out)
    assert ok and ok_ref
    got = out.cpu().numpy()
    assert (got[batch * dim:] == 1).all(), "wrote past the output"
    np.testing.assert_array_equal(bits(got[:batch * dim]), bits(ref[:batch * dim]))


@pytest.mark.parametrize("bit_rate", [8, 4, 2])
@pytest.mark.parametrize("sb_last", [True, False])
@pytest.mark.parametrize("batch", [40, 1500])
def test_row_widths_and_alignments(gpu_ctx, oracle, bit_rate, sb_last, batch):
    """40 bags are partly for a block each (few_bags_kernel.cu), 1500 for a warp each."""
    rng = np.random.default_rng(100 * bit_rate + sb_last)
    for dim in (1, 2, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 150, 192, 193, 255, 256, 257, 300, 320, 321, 520, 1024):
        for pad in (0, 1, 2, 4):
            check(oracle, rng, bit_rate, dim, batch, sb_last, pad, weighted=(dim + pad) % 2 == 0)


@pytest.mark.parametrize("bit_rate", [8, 4, 2])
@pytest.mark.parametrize("batch", [7104, 7105, 28416, 56832, 56833])
def test_lanes_per_bag(gpu_ctx, oracle, bit_rate, batch):
    rng = np.random.default_rng(7 * bit_rate + batch)
    for dim in (20, 32, 64, 128):
        check(oracle, rng, bit_rate, dim, batch, dim != 64, 0)


@pytest.mark.parametrize("bit_rate", [8, 4])
@pytest.mark.parametrize("batch", [50, 2000])
def test_rows_beyond_4gb(gpu_ctx, oracle, bit_rate, batch):
    """Few rows, far apart: the table's pitch puts them beyond 32-bit offsets.  50 bags are for a block each, 2000 for a warp;
    then beside a small table in one launch."""
    rng = np.random.default_rng(bit_rate)
    dim, rows, stride = 64, 70_000, 65_536
    used = np.sort(rng.choice(rows, 64, replace=False))
    used[-1] = rows - 1
    compact = random_fused_table(rng, len(used), dim, bit_rate)
    table = torch.zeros(rows * stride, dtype=torch.uint8, device="cuda").view(rows, stride)
    table[torch.from_numpy(used).cuda(), :row_bytes(bit_rate, dim)] = dev(compact)
    lengths = rng.choice(EDGE_LENGTHS[-6:] if batch == 50 else EDGE_LENGTHS, batch)
    n = int(lengths.sum())
    pick = rng.integers(0, len(used), n)
    offsets = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    w = rng.standard_normal(n).astype(np.float32)
    ok_ref, ref = oracle.spmdm(bit_rate, dim, len(used), compact, pick, offsets, w, False, np.float32, False, True,
                               output_size=batch, index_size=n)
    out = torch.zeros(batch * dim, device="cuda")
    kern = generate(bit_rate, dim, True, True, stride)
    assert kern(batch, n, rows, table, dev(used[pick]), dev(offsets), dev(w), out) and ok_ref
    np.testing.assert_array_equal(bits(out.cpu().numpy()), bits(ref))
    out2, out3 = torch.zeros_like(out), torch.zeros_like(out)
    plan = F.MultiTablePlan([(kern, batch, n, rows, table, dev(used[pick]), dev(offsets), dev(w), out2, None),
                             (generate(bit_rate, dim, True, True, -1), batch, n, len(used), dev(compact), dev(pick), dev(offsets),
                              dev(w), out3, None)])
    plan.launch()
    assert F.status_read(0)[0]
    np.testing.assert_array_equal(bits(out2.cpu().numpy()), bits(ref))
    np.testing.assert_array_equal(bits(out3.cpu().numpy()), bits(ref))
    plan.close()
    bad = used[pick].copy()
    bad[0] = rows
    assert not kern(batch, n, rows, table, dev(bad), dev(offsets), dev(w), out)


def test_more_tables_than_one_launch_takes(gpu_ctx, oracle):
    rng = np.random.default_rng(9)
    calls, want = [], []
    for t in range(70):
        bit_rate, dim, batch, rows = (8, 4, 2)[t % 3], (64, 20, 300, 128)[t % 4], 33 + t, 50
        table = random_fused_table(rng, rows, dim, bit_rate)
        lengths = rng.choice(EDGE_LENGTHS, batch)
        n = int(lengths.sum())
        indices = rng.integers(0, rows, n)
        offsets = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
        w = rng.standard_normal(n).astype(np.float32)
        want.append(oracle.spmdm(bit_rate, dim, rows, table, indices, offsets, w, False, np.float32, False, True,
                                 output_size=batch, index_size=n)[1])
        calls.append((generate(bit_rate, dim, True, True, -1), batch, n, rows, dev(table), dev(indices), dev(offsets),
                      dev(w), torch.zeros(batch * dim, device="cuda"), None))
    plan = F.MultiTablePlan(calls)
    plan.launch()
    assert F.status_read(0)[0]
    for c, ref in zip(calls, want):
        np.testing.assert_array_equal(bits(c[8].cpu().numpy()), bits(ref))
    plan.close()


@pytest.mark.parametrize("cols", [4, 7, 8, 33, 64, 100, 129, 256, 300, 512, 520, 1024, 1032, 2052])
def test_quantizer_blocks(gpu_ctx, oracle, cols):
    """Widths around the choices of rows per block and lanes per row, row counts around a block, and tables that start
    off a 16-byte boundary."""
    rng = np.random.default_rng(cols)
    for rows in (1, 17, 300):
        x = rng.standard_normal((rows, cols)).astype(np.float32)
        x[0] = 1.5  # no range
        for off in (0, 1):
            src = torch.empty(rows * cols + 4, device="cuda")[off:off + rows * cols].view(rows, cols)
            src.copy_(torch.from_numpy(x))
            out = torch.empty(rows * (cols + 8) + 8, dtype=torch.uint8, device="cuda")[off:off + rows * (cols + 8)]
            got = F.FloatToFused8BitRowwiseQuantizedSBFloat(src, out.view(rows, cols + 8)).cpu().numpy()
            np.testing.assert_array_equal(got, oracle.quantize_8bit(x))
        for b in (4, 2):
            if cols % (8 // b) == 0:
                got = F.FloatToFusedNBitRowwiseQuantizedSBHalf(b, dev(x)).cpu().numpy()
                np.testing.assert_array_equal(got, oracle.quantize_nbit(b, x))


@pytest.mark.parametrize("dim,out_dt,weighting", [(128, np.float32, "unweighted"), (64, np.float16, "weighted"),
                                                  (86, np.float16, "weighted"), (128, np.float32, "positional")])
def test_pageable_calls_in_parts(gpu_ctx, oracle, dim, out_dt, weighting):
    """Host arrays large enough to go up, through the lookup and down in parts of consecutive bags, some of them without
    any index; calls whose offsets do not cover the indices, or step back, return false."""
    rng = np.random.default_rng(dim)
    rows, batch = 3000, 30_001
    table = random_fused_table(rng, rows, dim, 8)
    lengths = rng.integers(0, 30, batch)
    lengths[5000:20000] = 0
    n = int(lengths.sum())
    indices = rng.integers(0, rows, n)
    offsets = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    w = rng.standard_normal(n).astype(np.float32)
    positional = weighting == "positional"
    kern = F.GenerateEmbeddingSpMDMWithStrides(dim, weighting != "unweighted", True, 16, positional, True,
                                               index_dtype=np.int64, offset_dtype=np.int64, out_dtype=out_dt)
    ok_ref, ref = oracle.spmdm(8, dim, rows, table, indices, offsets, w if weighting != "unweighted" else None, True, out_dt,
                               positional, True, output_size=batch, index_size=n)
    out = np.zeros(batch * dim, dtype=out_dt)
    gpu_ctx.register_table(table)
    for _ in range(2):
        out[:] = 0
        assert kern(batch, n, rows, table, indices, offsets, w, out) and ok_ref
        np.testing.assert_array_equal(bits(out), bits(ref[:batch * dim]))
    for bad in (n - 1, n + 1):
        o = offsets.copy()
        o[-1] = bad
        assert not kern(batch, n, rows, table, indices, o, w, out)
    o = offsets.copy()
    o[batch // 2] = n
    assert not kern(batch, n, rows, table, indices, o, w, out)
    i = indices.copy()
    i[n // 2] = rows
    assert not kern(batch, n, rows, table, i, offsets, w, out)
    assert kern(batch, n, rows, table, indices, offsets, w, out)
    np.testing.assert_array_equal(bits(out), bits(ref[:batch * dim]))
    gpu_ctx.unregister_table(table)


@pytest.mark.parametrize("batch", [1, 3, 33, 5000, 12_288, 12_289])
def test_lengths_without_a_scan(gpu_ctx, oracle, batch):
    rng = np.random.default_rng(batch)
    rows, dim = 400, 64
    table = random_fused_table(rng, rows, dim, 4)
    lengths = rng.integers(0, 6, batch)
    lengths[rng.integers(0, batch, 3)] = 40
    n = int(lengths.sum())
    indices = rng.integers(0, rows, n).astype(np.int32)
    w = rng.standard_normal(n).astype(np.float32)
    for odt in (np.int32, np.int64):
        kern = F.GenerateEmbeddingSpMDMNBit(4, dim, True, True, use_offsets=False, index_dtype=np.int32, offset_dtype=odt)
        ok_ref, ref = oracle.spmdm(4, dim, rows, table, indices, lengths.astype(odt), w, True, np.float32, False, False,
                                   output_size=batch, index_size=n)
        out = torch.zeros(batch * dim, device="cuda")
        args = (dev(table), dev(indices), dev(lengths.astype(odt)), dev(w), out)
        assert kern(batch, n, rows, *args) and ok_ref
        np.testing.assert_array_equal(bits(out.cpu().numpy()), bits(ref))
        assert not kern(batch, n - 1, rows, *args)       # the lengths do not add up to index_size


@pytest.mark.parametrize("batch", [10_656, 10_657, 21_312, 21_313])
def test_pruned_launches_around_what_fits_the_chip(gpu_ctx, oracle, batch):
    rng = np.random.default_rng(batch)
    kept, full, dim = 400, 900, 128
    table = random_fused_table(rng, kept, dim, 2)
    mapping = np.full(full, -1, dtype=np.int32)
    mapping[rng.choice(full, kept, replace=False)] = np.arange(kept, dtype=np.int32)
    lengths = rng.integers(0, 4, batch)
    lengths[rng.integers(0, batch, 60)] = rng.choice(EDGE_LENGTHS, 60)
    offsets = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    indices = rng.integers(0, full, offsets[-1]).astype(np.int64)
    kern = F.GenerateEmbeddingSpMDMNBitRowWiseSparse(2, dim, False, True, index_dtype=np.int64, offset_dtype=np.int32)
    ok_ref, ref = oracle.spmdm_rowwise_sparse(2, dim, full, table, indices, mapping, offsets, None, True)
    out = torch.zeros(batch * dim, device="cuda")
    assert kern(batch, len(indices), full, dev(table), dev(indices), dev(offsets), None, out, dev(mapping)) and ok_ref
    np.testing.assert_array_equal(bits(out.cpu().numpy()), bits(ref))
