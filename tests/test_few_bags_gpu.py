"""Lookups of a handful of bags, which have a kernel of their own (a block per bag and 128 columns, few_bags_rule.h says up to
how many), at its edges: the 256 rows that a block resolves at a time, the 128 columns of a tile, rows that words cannot
copy, and the batches and average lengths at which the other kernels take over, with those kernels at the same widths,
alignments and options just beyond.  Bit for bit against the CPU oracle."""
import numpy as np
import pytest
import torch

import fbgemm_b200 as F
from conftest import bits
from helpers import mapping_table, random_fused_table

pytestmark = pytest.mark.gpu
LENGTHS = np.array([0, 1, 2, 31, 32, 33, 255, 256, 257, 511, 513])


def dev(a):
    return None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()


OUT = {"f32": (np.float32, torch.float32), "f16": (np.float16, torch.float16), "bf16": (np.uint16, torch.bfloat16)}


def sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


def check(oracle, rng, bit_rate, dim, batch, sb_last=True, pad=0, weighted=True, positional=False, use_offsets=True, mean=False,
          index=np.int64, offset=np.int32, out="f32", lengths=None, bad=False):
    rows = 300
    stride = (dim * bit_rate + 7) // 8 + (8 if bit_rate == 8 and sb_last else 4) + pad
    table = random_fused_table(rng, rows, dim, bit_rate, stride, not sb_last)
    lengths = rng.choice(LENGTHS if lengths is None else lengths, batch)
    n = int(lengths.sum())
    indices = rng.integers(0, rows, n).astype(index)
    if not sb_last:
        indices[rng.random(n) < 0.3] = -1
    if bad and n:
        indices[rng.integers(0, n)] = rows
    offsets = np.concatenate([[0], np.cumsum(lengths)]).astype(offset)
    ol = offsets if use_offsets else lengths.astype(offset)
    w = rng.standard_normal(n).astype(np.float32) if weighted else None
    ok_ref, ref = oracle.spmdm_ex(bit_rate, dim, rows, table, indices, ol, w, mean, out, positional, use_offsets, -1, stride, sb_last,
                                  False, output_size=batch, index_size=n)
    kw = dict(index_dtype=index, offset_dtype=offset, out_dtype=OUT[out][0], is_bf16_out=out == "bf16")
    if bit_rate == 8:
        kern = F.GenerateEmbeddingSpMDMWithStrides(dim, weighted, mean, 16, positional, use_offsets, -1, stride, sb_last, **kw)
    else:
        kern = F.GenerateEmbeddingSpMDMNBitWithStrides(bit_rate, dim, weighted, mean, 16, positional, use_offsets, -1, stride, sb_last, **kw)
    res = torch.ones(batch * dim + 8, dtype=OUT[out][1], device="cuda")
    args = (batch, n, rows, dev(table), dev(indices), dev(ol), dev(w), res)
    assert bool(kern(*args)) == bool(ok_ref) == (not (bad and n))
    assert (res[batch * dim:] == 1).all(), "wrote past the output"
    if ok_ref:
        got = res.view(torch.int32 if out == "f32" else torch.int16).cpu().numpy()
        np.testing.assert_array_equal(got[:batch * dim], bits(ref[:batch * dim]).view(got.dtype))
    else:   # the record names the index
        kern.launch(*args, slot=7)
        ok, info = F.status_read(7)
        at = int(np.flatnonzero(indices == rows)[0])
        assert not ok and info == [1, int(np.searchsorted(offsets, at, "right")) - 1, at, rows]


@pytest.mark.parametrize("bit_rate", [8, 4, 2])
@pytest.mark.parametrize("sb_last", [True, False])
def test_widths_and_alignments(gpu_ctx, oracle, bit_rate, sb_last):
    rng = np.random.default_rng(10 * bit_rate + sb_last)
    for dim in (1, 4, 20, 64, 86, 127, 128, 129, 256, 300, 1024):
        for pad in (0, 1, 2, 4):
            check(oracle, rng, bit_rate, dim, 7, sb_last, pad)
            check(oracle, rng, bit_rate, dim, 4 * sms() + 8, sb_last, pad, lengths=np.array([0, 1, 5, 33]))


@pytest.mark.parametrize("bit_rate", [8, 4, 2])
def test_options(gpu_ctx, oracle, bit_rate):
    rng = np.random.default_rng(bit_rate)
    pick = lambda *x: x[rng.integers(len(x))]  # noqa: E731
    # a block per bag, then a warp
    for batches, lengths in (((1, 3, 60), None), ((1300, 2500), np.array([0, 1, 5, 33]))):
        for k in range(16):
            check(oracle, rng, bit_rate, pick(32, 64, 100, 256), pick(*batches), pick(True, False), 0, weighted=k % 2 == 0,
                  positional=k % 4 == 0, use_offsets=k % 3 != 0, mean=pick(True, False), index=pick(np.int32, np.int64),
                  offset=pick(np.int32, np.int64), out=pick("f32", "f16", "bf16"), lengths=lengths)
        check(oracle, rng, bit_rate, 64, batches[1], bad=True, lengths=lengths)


@pytest.mark.parametrize("use_offsets", [True, False])
def test_batches_around_the_change(gpu_ctx, oracle, use_offsets):
    rng = np.random.default_rng(4)
    n = sms()
    for more in (-1, 0, 1):
        check(oracle, rng, 8, 64, 4 * n + more, use_offsets=use_offsets, lengths=np.array([33, 40]))       # four blocks an SM
        check(oracle, rng, 8, 64, 8 * n + more, use_offsets=use_offsets, lengths=np.array([61, 70]))       # eight of long bags
        check(oracle, rng, 4, 256, 2 * n + more, use_offsets=use_offsets, lengths=np.array([25, 40]))      # in two tiles
        check(oracle, rng, 8, 86, 2 * n + more, use_offsets=use_offsets, lengths=np.array([20, 29]))       # by halves
    for bit_rate, dim, average in ((8, 64, 32), (4, 64, 20), (8, 86, 20), (4, 129, 16), (8, 129, 60)):
        for length in (average - 1, average):
            check(oracle, rng, bit_rate, dim, 50, use_offsets=use_offsets, lengths=np.array([length]))


@pytest.mark.parametrize("bit_rate", [8, 4, 2])
def test_pruned_and_unlike_sizes(gpu_ctx, oracle, bit_rate):
    rng = np.random.default_rng(20 + bit_rate)
    dim, batch, rows = 100, 9, 400
    cit, dense = mapping_table(rng, rows, 0.5)
    table = random_fused_table(rng, max(dense, 1), dim, bit_rate)
    lengths = rng.choice(LENGTHS, batch)
    n = int(lengths.sum())
    indices = rng.integers(0, rows, n)
    offsets = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    w = rng.standard_normal(n).astype(np.float32)
    ok_ref, ref = oracle.spmdm_rowwise_sparse(bit_rate, dim, rows, table, indices, cit, offsets, w, False)
    kw = dict(index_dtype=np.int64, offset_dtype=np.int32)
    kern = (F.GenerateEmbeddingSpMDMRowWiseSparse(dim, True, False, **kw) if bit_rate == 8
            else F.GenerateEmbeddingSpMDMNBitRowWiseSparse(bit_rate, dim, True, False, **kw))
    out = torch.zeros(batch * dim, device="cuda")
    args = [dev(table), dev(indices), dev(offsets), dev(w), out, dev(cit)]
    assert kern(batch, n, rows, *args) and ok_ref
    np.testing.assert_array_equal(bits(out.cpu().numpy()), bits(ref))
    assert not kern(batch, n + 1, rows, *args)      # offsets that do not add up to index_size
    args[2] = dev(offsets[::-1].copy())             # that step backwards
    assert not kern(batch, n, rows, *args)
    args[2] = dev(offsets)
    assert kern(batch, n, rows, *args)              # and the next call is clean
