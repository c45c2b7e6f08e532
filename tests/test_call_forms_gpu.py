"""Forms of the calls that the common case does not use: tables and index arrays
in page-locked host memory, pruning maps into larger tables, output rows farther
apart than their columns, operators whose tables change or that are copied, and
calls that overlap on several streams.  Bit for bit against the CPU oracle."""
import copy
import ctypes as C

import numpy as np
import pytest
import torch

import fbgemm_b200 as F
from fbgemm_b200 import _capi, tbe
from fbgemm_b200 import embedding as E
from conftest import bits
from helpers import build_op_inputs, oracle_op_forward, random_fused_table, random_plain_table, row_bytes

pytestmark = pytest.mark.gpu
ST = tbe.SparseType


def dev(a):
    return None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()


def bags(rng, batch, rows, hi=40):
    lengths = rng.integers(0, hi, batch)
    offsets = np.concatenate([[0], np.cumsum(lengths)])
    n = int(offsets[-1])
    return n, rng.integers(0, rows, n).astype(np.int64), offsets.astype(np.int64)


# ---- page-locked host memory ---------------------------------------------------

@pytest.mark.parametrize("call", ["awaited", "launch"])
def test_arrays_in_page_locked_memory(gpu_ctx, oracle, call):
    """The GPU reads page-locked arrays where they lie: a table tensor, and index arrays as the numpy views of pinned
    tensors."""
    rng = np.random.default_rng(1)
    rows, dim, batch = 200, 64, 33
    table = random_fused_table(rng, rows, dim, 8)
    n, indices, offsets = bags(rng, batch, rows)
    ok_ref, ref = oracle.spmdm(8, dim, rows, table, indices, offsets, None, False, np.float32)
    assert ok_ref
    k = F.GenerateEmbeddingSpMDM(dim, False, False, index_dtype=np.int64, offset_dtype=np.int64)
    pinned = [torch.from_numpy(a).pin_memory() for a in (table, indices, offsets)]
    forms = [pinned, [dev(table), pinned[1].numpy(), pinned[2].numpy()], [pinned[0], dev(indices), pinned[2].numpy()]]
    for t, i, o in forms:
        out = torch.ones(batch * dim, device="cuda")
        if call == "awaited":
            assert k(batch, n, rows, t, i, o, None, out)
        else:
            k.launch(batch, n, rows, t, i, o, None, out, slot=40)
            assert F.status_read(40)[0]
        np.testing.assert_array_equal(bits(out.cpu().numpy()), bits(ref[:batch * dim]))


def test_pageable_arrays_are_refused_beside_device_arrays(gpu_ctx):
    rng = np.random.default_rng(2)
    rows, dim, batch = 50, 32, 4
    table = random_fused_table(rng, rows, dim, 8)
    n, indices, offsets = bags(rng, batch, rows)
    k = F.GenerateEmbeddingSpMDM(dim, False, False, index_dtype=np.int64, offset_dtype=np.int64)
    out = torch.empty(batch * dim, device="cuda")
    for call in (k, k.launch):
        with pytest.raises(Exception):
            call(batch, n, rows, dev(table), indices, dev(offsets), None, out)
        with pytest.raises(Exception):
            call(batch, n, rows, torch.from_numpy(table), dev(indices), dev(offsets), None, out)


# ---- sequence rows with room between them ----------------------------------------

@pytest.mark.parametrize("D,n", [(16, 32), (16, 45), (10, 40), (128, 33)])
@pytest.mark.parametrize("filled", [False, True])
def test_sequence_rows_keep_what_lies_between_them(gpu_ctx, D, n, filled):
    """A pruned row (-1) is D columns of zeros; the bytes up to the next row are the caller's, whatever the rows around
    it.  Only the filled form clears rows that nothing names, in full."""
    rng = np.random.default_rng(D + n)
    rows, pitch_cols = 50, D + 8
    stride = tbe.padded_row_size_in_bytes(D, ST.INT8, 4, 4)
    table = random_fused_table(rng, rows, D, 8, stride, True)
    idx = rng.integers(0, rows, n).astype(np.int32)
    idx[rng.permutation(n)[:n // 3]] = -1
    idx[n - 2] = rows + 5                              # out of range: reported, and left alone (filled: cleared)
    op = tbe.IntNBitSequenceEmbedding(dev(table.reshape(-1)), np.zeros(1, np.int64), np.array([int(ST.INT8)], np.uint8), D, 4,
                                      ST.FP32, False)
    out = torch.full((n, pitch_cols), 7.0, device="cuda")
    d_idx, d_off = dev(idx), dev(np.array([0, n], np.int32))
    fn = _capi.lib().fbgemm_b200_sequence_lookup_filled if filled else _capi.lib().fbgemm_b200_sequence_lookup
    rc = fn(gpu_ctx.handle, op.dev_weights.data_ptr(), op._desc.data_ptr(), 1, 1, D, d_idx.data_ptr(), d_off.data_ptr(), 4, n,
            out.data_ptr(), op.out_code, 4 * pitch_cols, 0, 4, 7, 41, torch.cuda.current_stream().cuda_stream)
    _capi.check(rc, "sequence lookup")
    assert not F.status_read(41)[0]
    got = out.cpu().numpy()
    sb = table[:, :4].copy().view(np.float16).astype(np.float32)
    for k in range(n):
        if idx[k] == -1:
            want = np.zeros(D, np.float32)
        elif idx[k] >= rows:
            want = np.full(D, 0.0 if filled else 7.0, np.float32)
        else:
            q = table[idx[k], 4:4 + D].astype(np.float64)
            want = (np.float64(sb[idx[k], 0]) * q + np.float64(sb[idx[k], 1])).astype(np.float32)
        np.testing.assert_array_equal(got[k, :D], want, err_msg=f"row {k}")
        if not (filled and idx[k] >= rows):
            assert (got[k, D:] == 7.0).all(), f"row {k}: bytes between the rows were written"


# ---- pruning maps into larger tables -------------------------------------------------

BIG = (1 << 32) + (300 << 20)   # bytes of the table


@pytest.fixture(scope="module")
def big_table():
    yield torch.zeros(BIG, dtype=torch.uint8, device="cuda")
    torch.cuda.empty_cache()


@pytest.mark.parametrize("fmt", [8, 4, 2, "f32", "f16"])
@pytest.mark.parametrize("batch", [40, 20_000, 60_000])
@pytest.mark.parametrize("weights", [None, "per_index", "positional"])
def test_pruning_map_into_a_table_beyond_4gb(gpu_ctx, oracle, big_table, fmt, batch, weights):
    """The map is short, the table that it names rows of is not: rows on both sides of 4 GB, and the two next to it."""
    rng = np.random.default_rng(batch + len(str(weights)))
    dim = 128 if batch > 40 else 100
    used_n, map_rows = 64, 300
    quantized = fmt in (8, 4, 2)
    compact = random_fused_table(rng, used_n, dim, fmt) if quantized else random_plain_table(rng, used_n, dim, fmt)
    raw = compact.view(np.uint8).reshape(used_n, -1)
    stride = raw.shape[1]
    total = BIG // stride
    edge = (1 << 32) // stride
    used = np.unique(np.concatenate([[0, edge - 2, edge - 1, edge, edge + 1, total - 1],
                                     rng.choice(total, 2 * used_n, replace=False)]))
    used = np.sort(np.concatenate([rng.permutation(np.setdiff1d(used, [0, edge - 2, edge - 1, edge, edge + 1, total - 1]))[:used_n - 6],
                                   [0, edge - 2, edge - 1, edge, edge + 1, total - 1]]))
    big = big_table[:total * stride].view(total, stride)
    big[torch.from_numpy(used).cuda()] = dev(raw)
    to_compact = rng.integers(-1, used_n, map_rows).astype(np.int32)
    to_big = np.where(to_compact >= 0, used[to_compact], -1).astype(np.int32)
    lengths = rng.integers(0, 70, batch) if batch == 40 else rng.integers(0, 4, batch)
    offsets = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    n = int(offsets[-1])
    indices = rng.integers(0, map_rows, n).astype(np.int64)
    positional = weights == "positional"
    w = None if weights is None else rng.standard_normal(80 if positional else n).astype(np.float32)
    kw = dict(index_dtype=np.int64, offset_dtype=np.int32)
    if quantized:
        ok_ref, ref = oracle.spmdm_rowwise_sparse(fmt, dim, map_rows, compact, indices, to_compact, offsets, w, False, positional)
        gen = ((lambda *a: F.GenerateEmbeddingSpMDMRowWiseSparse(*a, **kw)) if fmt == 8
               else (lambda *a: F.GenerateEmbeddingSpMDMNBitRowWiseSparse(fmt, *a, **kw)))
    else:
        ok_ref, ref = oracle.spmdm_plain_rowwise_sparse(fmt, dim, map_rows, compact, indices, to_compact, offsets, w, False,
                                                        positional)
        gen = lambda *a: F.GenerateEmbeddingSpMDMRowWiseSparse(  # noqa: E731
            *a, in_dtype=np.float32 if fmt == "f32" else np.float16, **kw)
    assert ok_ref
    k = gen(dim, w is not None, False, 16, positional)
    out = torch.ones(batch * dim, device="cuda")
    assert k(batch, n, map_rows, big, dev(indices), dev(offsets), dev(w), out, dev(to_big))
    big[torch.from_numpy(used).cuda()] = 0
    np.testing.assert_array_equal(bits(out.cpu().numpy()), bits(ref[:batch * dim]))


def test_pruning_maps_beside_other_tables_in_one_plan(gpu_ctx, oracle, big_table):
    """Tables with and without a map, with rows on both sides of 4 GB, in one call."""
    rng = np.random.default_rng(11)
    dim, batch, rows, used_n = 128, 50, 200, 40
    kw = dict(index_dtype=np.int64, offset_dtype=np.int32)
    calls, checks = [], []
    for t, fmt in enumerate((8, 4, 2, 4)):
        compact = random_fused_table(rng, used_n, dim, fmt)
        stride = compact.shape[1]
        total, edge = BIG // stride, (1 << 32) // stride
        used = np.unique(np.concatenate([[edge - 2, edge - 1, edge, edge + 1, total - 1 - t], t + 4 * rng.choice(total // 8, used_n - 5, replace=False)]))
        compact = compact[:len(used)]
        table = torch.zeros(1, dtype=torch.uint8)
        if fmt != 4:
            big_table.zero_() if t == 0 else None
            table = big_table[:total * stride].view(total, stride) if t == 0 else torch.zeros((total, stride), dtype=torch.uint8, device="cuda")
            table[torch.from_numpy(used).cuda()] = dev(compact)
        n, indices, offsets = bags(rng, batch, rows)
        offsets = offsets.astype(np.int32)
        out = torch.ones(batch * dim, device="cuda")
        if fmt == 4:      # no map
            table, rows_of = dev(compact), len(used)
            indices = indices % rows_of
            ok_ref, ref = oracle.spmdm(4, dim, rows_of, compact, indices, offsets, None, False, np.float32)
            k, cit = F.GenerateEmbeddingSpMDMNBit(4, dim, False, False, **kw), None
        else:
            rows_of, to_compact = rows, rng.integers(-1, len(used), rows).astype(np.int32)
            ok_ref, ref = oracle.spmdm_rowwise_sparse(fmt, dim, rows, compact, indices, to_compact, offsets)
            k = (F.GenerateEmbeddingSpMDMRowWiseSparse(dim, False, False, **kw) if fmt == 8
                 else F.GenerateEmbeddingSpMDMNBitRowWiseSparse(fmt, dim, False, False, **kw))
            cit = dev(np.where(to_compact >= 0, used[to_compact], -1).astype(np.int32))
        assert ok_ref
        calls.append((k, batch, n, rows_of, table, dev(indices), dev(offsets), None, out, cit))
        checks.append((out, ref))
    plan = F.MultiTablePlan(calls, 0, slot=45)
    plan.launch()
    assert F.status_read(45)[0]
    for out, ref in checks:
        np.testing.assert_array_equal(bits(out.cpu().numpy()), bits(ref[:batch * dim]))


# ---- the tables of an operator -------------------------------------------------------

def small_op(rng, tys=(ST.INT8, ST.INT4, ST.FP16), rows=(60, 50, 40), dims=(16, 32, 8), B=9, idt=np.int32):
    tables, blob, w_off, D_off, offsets, indices, _ = build_op_inputs(rng, tys, dims, rows, B, 6, 4, False, idt)
    op = tbe.IntNBitTableBatchedEmbeddingBags(dev(blob), w_off, np.array([int(t) for t in tys], np.uint8), D_off,
                                              int(D_off[-1]), tbe.PoolingMode.SUM, 4, ST.FP32, False)
    def want(oracle, blob=blob):
        return oracle_op_forward(oracle, tys, dims, rows, blob, w_off, D_off, indices, offsets, None, B, False, 0, False, 4)
    return op, blob, w_off, tables, dev(indices), dev(offsets), want


def result(op, indices, offsets):
    out = op.forward(indices, offsets, slot=42)
    assert F.status_read(42)[0]
    return out.cpu().numpy().view(np.uint32)


def test_a_table_set_of_a_closed_context_is_refused(gpu_ctx):
    rng = np.random.default_rng(5)
    op, _, _, _, indices, offsets, _ = small_op(rng)
    ctx = E.Context(0)
    calls = (_capi.TableCall * op.T)()
    columns = (C.c_int64 * op.T)(*[int(c) for c in op.D_offsets[:-1]])
    for t in range(op.T):
        calls[t].cfg, calls[t].data_size, calls[t].input = op.kernels[t].cfg, op.rows[t], op.tables[t].data_ptr()
    sets = []
    for _ in range(3):
        h = C.c_void_p()
        _capi.check(_capi.lib().fbgemm_b200_table_set_create(ctx.handle, calls, columns, op.T, C.byref(h)), "create")
        sets.append(h)
    out = torch.empty((9, op.total_D), device="cuda")
    args = (9, indices.data_ptr(), indices.numel(), offsets.data_ptr(), None, out.data_ptr(), 0, None)
    assert _capi.lib().fbgemm_b200_table_set_forward(sets[0], *args) == 0
    torch.cuda.synchronize()
    _capi.lib().fbgemm_b200_table_set_destroy(sets[1])   # before its context ...
    ctx.close()
    assert _capi.lib().fbgemm_b200_table_set_forward(sets[0], *args) == _capi.EINVAL
    for h in (sets[0], sets[2]):                         # ... and after it
        _capi.lib().fbgemm_b200_table_set_destroy(h)


# ---- operators whose tables change, or that have none ---------------------------------

def test_a_table_put_in_place_of_another_is_read(gpu_ctx, oracle):
    rng = np.random.default_rng(3)
    op, blob, w_off, tables, indices, offsets, want = small_op(rng)
    np.testing.assert_array_equal(result(op, indices, offsets), want(oracle))
    other = random_fused_table(rng, tables[1].shape[0], 32, 4, tables[1].shape[1], True)
    op.tables[1] = dev(other.reshape(-1))
    changed = blob.copy()
    changed[int(w_off[1]):int(w_off[2])] = other.reshape(-1)
    np.testing.assert_array_equal(result(op, indices, offsets), want(oracle, changed))
    op.tables = [dev(blob[int(a):int(b)]) for a, b in zip(w_off, list(w_off[1:]) + [len(blob)])]
    np.testing.assert_array_equal(result(op, indices, offsets), want(oracle))


def test_operators_without_tables_and_with_empty_ones(gpu_ctx):
    op = tbe.IntNBitTableBatchedEmbeddingBags(torch.zeros(0, dtype=torch.uint8, device="cuda"), [], [], [0], 0)
    assert op.T == 0
    # one table without rows: bags without indices pool to zeros
    op = tbe.IntNBitTableBatchedEmbeddingBags(torch.zeros(0, dtype=torch.uint8, device="cuda"), [0], [int(ST.INT8)], [0, 16],
                                              16, output_dtype=ST.FP32)
    out = op.forward(torch.zeros(0, dtype=torch.int32, device="cuda"), torch.zeros(6, dtype=torch.int32, device="cuda"), slot=43)
    assert F.status_read(43)[0] and out.shape == (5, 16) and (out.cpu() == 0).all()


# ---- copies of an operator -------------------------------------------------------------

def test_copies_of_an_operator_have_tables_of_their_own(gpu_ctx, oracle):
    rng = np.random.default_rng(4)
    op, blob, w_off, tables, indices, offsets, want = small_op(rng)
    ref = want(oracle)
    np.testing.assert_array_equal(result(op, indices, offsets), ref)
    shallow, deep = copy.copy(op), copy.deepcopy(op)
    op.dev_weights.zero_()          # the deep copy's tables are its own
    np.testing.assert_array_equal(result(deep, indices, offsets), ref)
    op.dev_weights.copy_(dev(blob))
    del op
    np.testing.assert_array_equal(result(shallow, indices, offsets), ref)
    del shallow
    np.testing.assert_array_equal(result(deep, indices, offsets), ref)
    k = copy.deepcopy(deep.kernels[0])
    assert C.addressof(k.cfg) != C.addressof(deep.kernels[0].cfg)


# ---- overlapping calls of one table ----------------------------------------------------

@pytest.mark.parametrize("bit_rate,dim,batch", [(8, 128, 1000), (8, 86, 301), (8, 128, 4096), (4, 64, 700),
                                                (4, 33, 4096), (4, 64, 4096), (2, 128, 1024), (2, 128, 4096), (2, 112, 2500),
                                                (2, 100, 4096)])
@pytest.mark.parametrize("pruned", [False, True])
def test_calls_that_overlap_on_several_streams(gpu_ctx, oracle, bit_rate, dim, batch, pruned):
    """Which kernel takes a call depends on what runs beside it; the rows do not."""
    rng = np.random.default_rng(bit_rate * dim + batch)
    rows, calls = 500, 40
    table = random_fused_table(rng, rows, dim, bit_rate)
    cit = np.where(rng.random(rows) < 0.4, -1, rng.permutation(rows)).astype(np.int32) if pruned else None
    n, indices, offsets = bags(rng, batch, rows, 70)
    if pruned:
        ok_ref, ref = oracle.spmdm_rowwise_sparse(bit_rate, dim, rows, table, indices, cit, offsets, None, True)
        k = (F.GenerateEmbeddingSpMDMRowWiseSparse(dim, False, True, index_dtype=np.int64, offset_dtype=np.int64) if bit_rate == 8
             else F.GenerateEmbeddingSpMDMNBitRowWiseSparse(bit_rate, dim, False, True, index_dtype=np.int64, offset_dtype=np.int64))
    else:
        ok_ref, ref = oracle.spmdm(bit_rate, dim, rows, table, indices, offsets, None, True, np.float32)
        k = (F.GenerateEmbeddingSpMDM(dim, False, True, index_dtype=np.int64, offset_dtype=np.int64) if bit_rate == 8
             else F.GenerateEmbeddingSpMDMNBit(bit_rate, dim, False, True, index_dtype=np.int64, offset_dtype=np.int64))
    assert ok_ref
    args = (dev(table), dev(indices), dev(offsets), None)
    outs = torch.ones(calls, batch * dim, device="cuda")
    d_cit = (dev(cit),) if pruned else ()
    streams = [torch.cuda.Stream() for _ in range(16)]
    torch.cuda.synchronize()
    for c in range(calls):          # one stream first, then all of them, then one again
        s = streams[c % 16 if 8 <= c < 32 else 0]
        k.launch(batch, n, rows, *args, outs[c], *d_cit, slot=44, stream=s.cuda_stream)
    torch.cuda.synchronize()
    assert F.status_read(44)[0]
    want = bits(ref[:batch * dim])
    for c in range(calls):
        np.testing.assert_array_equal(bits(outs[c].cpu().numpy()), want, err_msg=f"call {c}")
