"""Parity of the CUDA lookup with the CPU oracle, on the reference's own test grids
(bench/tbe_inference/.../test_int_nbit_split_embedding_codegen_lookup_function.py:372-487) extended
to every weight type, plus the edge cases of the domain (empty bags, pruned indices, ragged
bags, unaligned rows, very wide rows)."""
import random
import zlib

import numpy as np
import pytest

import oracle as O
from helpers import Case, assert_close, gpu_lookup, make_case, oracle_lookup

pytestmark = pytest.mark.gpu

ALIGN = {O.FP32: 1, O.FP16: 2, O.INT8: 4, O.INT4: 8, O.INT2: 16, O.FP8: 4}
OUT_ALIGN = {O.FP32: 1, O.FP16: 2, O.BF16: 2}


def seed_of(*args):
    return zlib.crc32(repr(args).encode()) & 0x7fffffff


def round_up(a, b):
    return (a + b - 1) // b * b


def run(c: Case, pooling, out_ty, what, fp8=(4, 7)):
    want = oracle_lookup(c, pooling, out_ty, fp8=fp8)
    got = gpu_lookup(c, pooling, out_ty, fp8=fp8)
    assert_close(got, want, out_ty, what)


@pytest.mark.parametrize("weights_ty", [O.INT8, O.INT4, O.FP16, O.FP8, O.FP32, O.INT2])
@pytest.mark.parametrize("pooling", [O.SUM, O.MEAN])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("index_dtype", [np.int32, np.int64])
@pytest.mark.parametrize("out_ty", [O.FP16, O.FP32, O.BF16])
@pytest.mark.parametrize("table_num", [1, 4, 10])
def test_random_multi_table_forward(weights_ty, pooling, weighted, index_dtype, out_ty, table_num):
    """Random tables: E in [1, 20000], D = 4*rand(1..1024) rounded to the type's alignment, B = 64,
    per-table bag length in [1, 100] (the reference's generator, :238-277)."""
    seed = seed_of(weights_ty, pooling, weighted, index_dtype.__name__, out_ty, table_num) & 0xffff
    rnd = random.Random(10000 + seed)
    rng = np.random.default_rng(10000 + seed)
    rows = [rnd.randint(1, 20000) for _ in range(table_num)]
    dims = [round_up(4 * rnd.randint(1, 1024), max(ALIGN[weights_ty], OUT_ALIGN[out_ty])) for _ in range(table_num)]
    if table_num == 10:
        dims = [min(d, 1024) for d in dims]   # keeps the CPU oracle quick; 4096-wide rows are covered below
    L = [rnd.randint(1, 100) for _ in range(table_num)]
    B = 64
    lens = np.concatenate([np.full(B, l) for l in L])
    c = make_case(rng, [weights_ty] * table_num, dims, rows, B, lens, index_dtype, weighted)
    run(c, pooling, out_ty, f"ty={weights_ty} dims={dims}")


BAG_TABLES = [
    [(1000, 16), (2000, 16)], [(2000, 256), (1000, 256)], [(2000, 512), (1000, 512)], [(2000, 1024), (1000, 1024)],
    [(2000, 2048), (1000, 2048)], [(2000, 4096), (1000, 4096)], [(2000, 16), (1000, 256)], [(2000, 16), (1000, 512)],
    [(2000, 16), (1000, 1024)], [(2000, 16), (1000, 2048)], [(2000, 16), (1000, 4096)],
]


@pytest.mark.parametrize("weights_ty", [O.INT8, O.FP8])
@pytest.mark.parametrize("pooling", [O.SUM, O.MEAN])
@pytest.mark.parametrize("weighted", [True, False])
@pytest.mark.parametrize("index_dtype", [np.int32, np.int64])
@pytest.mark.parametrize("out_ty", [O.FP16, O.FP32, O.BF16])
@pytest.mark.parametrize("tables", BAG_TABLES)
def test_double_table_forward_bag(weights_ty, pooling, weighted, index_dtype, out_ty, tables):
    """The reference's fixed two-table grid (:418-460), bag lengths 40 and 50, B = 64."""
    rng = np.random.default_rng(seed_of(weights_ty, pooling, weighted, out_ty, tables))
    rows = [e for e, _ in tables]
    dims = [d for _, d in tables]
    lens = np.concatenate([np.full(64, 40), np.full(64, 50)])
    c = make_case(rng, [weights_ty] * 2, dims, rows, 64, lens, index_dtype, weighted)
    run(c, pooling, out_ty, f"tables={tables}")


NOBAG_TABLES = [
    [(1000, 16), (2000, 16)], [(1000, 32), (2000, 32)], [(1000, 64), (2000, 64)], [(1000, 128), (2000, 128)],
    [(2000, 256), (1000, 256)], [(2000, 512), (1000, 512)], [(2000, 1024), (1000, 1024)],
    [(2000, 2048), (1000, 2048)], [(2000, 4096), (1000, 4096)],
]


@pytest.mark.parametrize("weights_ty", [O.INT8, O.INT4, O.FP8, O.FP16])
@pytest.mark.parametrize("out_ty", [O.FP16, O.FP32, O.BF16])
@pytest.mark.parametrize("index_dtype", [np.int32, np.int64])
@pytest.mark.parametrize("tables", NOBAG_TABLES)
def test_double_table_forward_nobag(weights_ty, out_ty, index_dtype, tables):
    """Pooling NONE, equal D across tables (:463-487)."""
    rng = np.random.default_rng(seed_of(weights_ty, out_ty, tables))
    rows = [e for e, _ in tables]
    dims = [d for _, d in tables]
    lens = np.concatenate([np.full(64, 40), np.full(64, 50)])
    c = make_case(rng, [weights_ty] * 2, dims, rows, 64, lens, index_dtype, False)
    run(c, O.NONE, out_ty, f"nobag tables={tables}")


@pytest.mark.parametrize("index_dtype", [np.int32, np.int64])
@pytest.mark.parametrize("out_ty", [O.FP32, O.FP16])
@pytest.mark.parametrize("pooling", [O.SUM, O.MEAN])
def test_mixed_types_jagged_empty_pruned(index_dtype, out_ty, pooling):
    """Mixed weight types in one launch, bag lengths uniform in [0, 200] (empty bags included),
    2% pruned (-1) indices, per-sample weights: the shape of benchmark configuration 5."""
    rng = np.random.default_rng(5)
    tys = [O.INT8, O.INT4, O.FP16, O.INT8, O.INT4, O.FP16, O.FP8, O.FP32, O.INT2]
    dims = [128, 128, 128, 64, 256, 32, 96, 20, 48]
    rows = [5000] * len(tys)
    B = 33
    lens = rng.integers(0, 201, len(tys) * B)
    lens[::7] = 0
    c = make_case(rng, tys, dims, rows, B, lens, index_dtype, True, prune_frac=0.02)
    run(c, pooling, out_ty, "mixed")


@pytest.mark.parametrize("weights_ty", [O.INT8, O.INT4, O.FP16, O.FP32, O.FP8, O.INT2])
@pytest.mark.parametrize("row_alignment", [1, 4, 16])
def test_row_alignment_and_unaligned_tables(weights_ty, row_alignment):
    """row_alignment 1 (unpadded rows, the layout upstream uses for CPU-built modules) and tables
    that start at odd byte offsets take the byte-wise path; results must not change."""
    rng = np.random.default_rng(row_alignment * 10 + weights_ty)
    dims = [round_up(d, ALIGN[weights_ty]) for d in (36, 128, 200)]
    c = make_case(rng, [weights_ty] * 3, dims, [777, 1000, 50], 16, [30, 5, 64], np.int64, True,
                  prune_frac=0.05, row_alignment=row_alignment, table_alignment=1 if row_alignment == 1 else 4)
    run(c, O.SUM, O.FP32, f"align={row_alignment}")


def test_all_bags_empty_through_c_abi():
    """No index at all: every output element must be zero.  (The operator, like the reference
    adapter, rejects an empty `indices`; the C ABI accepts it.)"""
    import torch
    from fbgemm_ascend_b200 import cabi

    rng = np.random.default_rng(0)
    c = make_case(rng, [O.INT8, O.FP16], [64, 32], [100, 100], 8, 0, np.int32)
    d = torch.device("cuda")
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(d)
    out = torch.full((8, 96), 7.0, dtype=torch.float16, device=d)
    cabi.lookup(t(c.dev_weights), t(c.weights_offsets), t(c.weights_tys), t(c.D_offsets), 96, 64,
                torch.zeros(0, dtype=torch.int32, device=d), t(c.offsets), O.SUM, out)
    assert float(out.abs().max()) == 0.0


def test_config1_full_size_matches_oracle_and_fbgemm():
    """Benchmark configuration 1 in full: T=1, E=100000, D=128 INT8 from N(0, 0.1) seed 0, B=512,
    L=20, int32, SUM, fp16 out -- against both the C restatement and the FBGEMM CPU kernels."""
    rng = np.random.default_rng(0)
    x = rng.normal(0.0, 0.1, (100_000, 128)).astype(np.float32)
    rows = O.pack_table(x, O.INT8)
    dev, wo, wt, do = O.concat_tables([rows], [O.INT8], [128])
    idx = rng.integers(0, 100_000, 512 * 20).astype(np.int32)
    offs = np.arange(0, 512 * 20 + 1, 20, dtype=np.int32)
    c = Case(dev, wo, wt, do, idx, offs, None, [O.INT8], [128], [100_000], 512)
    got = gpu_lookup(c, O.SUM, O.FP16)
    assert_close(got, oracle_lookup(c, O.SUM, O.FP16, impl="port"), O.FP16, "c1 vs port")
    assert_close(got, oracle_lookup(c, O.SUM, O.FP16, impl="ref"), O.FP16, "c1 vs fbgemm")


def test_error_flag_and_bad_arguments():
    import torch
    from fbgemm_ascend_b200 import cabi

    rng = np.random.default_rng(1)
    c = make_case(rng, [O.INT8], [32], [50], 4, 3, np.int64)
    c.indices[2] = -5   # invalid (only -1 means "pruned")
    d = torch.device("cuda")
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(d)
    flag = torch.zeros(1, dtype=torch.int32, device=d)
    out = torch.empty((4, 32), dtype=torch.float32, device=d)
    args = (t(c.dev_weights), t(c.weights_offsets), t(c.weights_tys), t(c.D_offsets), 32, 32, t(c.indices), t(c.offsets))
    cabi.lookup(*args, O.SUM, out, error_flag=flag)
    assert int(flag.item()) == 1
    c.indices[2] = -1
    assert_close(out.cpu().numpy(), oracle_lookup(c, O.SUM, O.FP32), O.FP32, "bad index skipped")
    with pytest.raises(RuntimeError, match="pooling_mode"):
        cabi.lookup(*args, 7, out)
    with pytest.raises(RuntimeError, match="rows_per_dest"):
        cabi.lookup(*args, O.SUM, out, dest_outputs=torch.zeros(1, dtype=torch.int64, device=d), rows_per_dest=0)
    # operator-level checks mirror the reference adapter's messages
    with pytest.raises(RuntimeError, match="indices can not be empty"):
        c2 = make_case(rng, [O.INT8], [32], [50], 4, 0, np.int64)
        gpu_lookup(c2, O.SUM, O.FP32)
    with pytest.raises(RuntimeError, match="is incorrect for feature count"):
        c3 = make_case(rng, [O.INT8, O.INT8], [32, 32], [50, 50], 4, 3, np.int64)
        c3.offsets = c3.offsets[:-1]
        gpu_lookup(c3, O.SUM, O.FP32)
    with pytest.raises(RuntimeError, match="Unsupported output_dtype"):
        gpu_lookup(c, O.SUM, 3)


def test_scatter_to_destinations_with_column_remap():
    """dest_outputs + output_col_offsets: the batch is split over several destination buffers and
    each table lands at a remapped column -- equal to lookup, split by rows, then permute."""
    import torch
    from fbgemm_ascend_b200 import cabi

    rng = np.random.default_rng(3)
    dims = [64, 128, 32, 128]
    c = make_case(rng, [O.INT8, O.INT4, O.FP16, O.INT8], dims, [300] * 4, 24, [20, 40, 3, 9], np.int64)
    want = oracle_lookup(c, O.SUM, O.FP16)
    perm = [2, 0, 3, 1]
    inv_dims = [dims[p] for p in perm]
    inv_off = np.concatenate([[0], np.cumsum(inv_dims)])
    off = np.concatenate([[0], np.cumsum(dims)])
    want_perm = np.concatenate([want[:, off[p]:off[p + 1]] for p in perm], axis=1)
    col = np.zeros(4, dtype=np.int64)
    for i, p in enumerate(perm):
        col[p] = inv_off[i]
    d = torch.device("cuda")
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(d)
    parts = [torch.zeros((8, sum(dims)), dtype=torch.float16, device=d) for _ in range(3)]
    ptrs = torch.tensor([p.data_ptr() for p in parts], dtype=torch.int64, device=d)
    cabi.lookup(t(c.dev_weights), t(c.weights_offsets), t(c.weights_tys), t(c.D_offsets), sum(dims), max(dims),
                t(c.indices), t(c.offsets), O.SUM, parts[0], output_col_offsets=t(col), dest_outputs=ptrs,
                rows_per_dest=8)
    got = torch.cat(parts, 0).float().cpu().numpy()
    assert_close(got, want_perm, O.FP16, "scatter+remap")


@pytest.mark.parametrize("weights_ty,D", [(O.INT8, 128), (O.INT4, 64), (O.FP16, 32), (O.INT8, 20)])
@pytest.mark.parametrize("pooling", [O.SUM, O.NONE])
def test_row_past_the_table_is_skipped_and_reported(weights_ty, D, pooling):
    """An index >= the table's row count is never dereferenced: with dev_weights_bytes known the row is
    treated like a pruned one (-1) and bit 4 of the error word is set.  Checked for a table in the
    middle of dev_weights (the row would belong to the next table) and for the last one (the row would
    lie outside the buffer)."""
    import torch
    from fbgemm_ascend_b200 import cabi

    rng = np.random.default_rng(11)
    E = [40, 30, 50]
    c = make_case(rng, [weights_ty] * 3, [D] * 3, E, 8, np.concatenate([np.full(8, 9), np.full(8, 12), np.full(8, 5)]), np.int64)
    offs = c.offsets
    bad_positions = [int(offs[8]) + 3, int(offs[16]) + 1, int(offs[23]) + 2]   # one in the middle table, two in the last
    for q in bad_positions:
        t = int(np.searchsorted(offs[::8], q, side="right") - 1)
        c.indices[q] = E[t] + (0 if q == bad_positions[0] else 1000)
    d = torch.device("cuda")
    t_ = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(d)
    flag = torch.zeros(1, dtype=torch.int32, device=d)
    n_out = c.indices.size if pooling == O.NONE else 8
    width = D if pooling == O.NONE else 3 * D
    out = torch.full((n_out, width), 3.0, dtype=torch.float32, device=d)
    cabi.lookup(t_(c.dev_weights), t_(c.weights_offsets), t_(c.weights_tys), t_(c.D_offsets), 3 * D, D, t_(c.indices),
                t_(c.offsets), pooling, out, error_flag=flag)
    assert int(flag.item()) == 4
    for q in bad_positions:
        c.indices[q] = -1
    assert_close(out.cpu().numpy(), oracle_lookup(c, pooling, O.FP32), O.FP32, "rows past the table pruned")


def test_offsets_that_disagree_with_the_index_count_are_reported():
    """offsets[T*B] != indices.numel() (the reference kernel asserts on it) sets bit 8; positions past
    `indices` are never read."""
    import torch
    from fbgemm_ascend_b200 import cabi

    rng = np.random.default_rng(12)
    c = make_case(rng, [O.INT8, O.INT8], [64, 64], [100, 100], 8, 6, np.int32)
    d = torch.device("cuda")
    t_ = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(d)
    flag = torch.zeros(1, dtype=torch.int32, device=d)
    out = torch.zeros((8, 128), dtype=torch.float16, device=d)
    short = c.indices[:-5]                      # offsets describe 5 more positions than there are indices
    cabi.lookup(t_(c.dev_weights), t_(c.weights_offsets), t_(c.weights_tys), t_(c.D_offsets), 128, 64, t_(short), t_(c.offsets),
                O.SUM, out, error_flag=flag)
    assert int(flag.item()) & 8
    flag.zero_()
    cabi.lookup(t_(c.dev_weights), t_(c.weights_offsets), t_(c.weights_tys), t_(c.D_offsets), 128, 64, t_(c.indices), t_(c.offsets),
                O.SUM, out, error_flag=flag)
    assert int(flag.item()) == 0
    assert_close(out.float().cpu().numpy(), oracle_lookup(c, O.SUM, O.FP16), O.FP16, "consistent offsets")


@pytest.mark.parametrize("out_dtype", ["float16", "float32"])
def test_scatter_with_rows_that_are_not_16_byte_aligned(out_dtype):
    """Destination scatter with an output row of 68 elements (136 or 272 bytes: alternate rows are
    misaligned for 16-byte stores), a batch that is not a multiple of the lane-group count, and bag lengths
    that differ a lot, so that bags straddle the lane groups' ranges."""
    import torch
    from fbgemm_ascend_b200 import cabi

    rng = np.random.default_rng(13)
    dims = [32, 16, 20]
    B = 13
    lens = rng.integers(0, 60, 3 * B)
    lens[5] = 300
    c = make_case(rng, [O.INT8, O.INT8, O.INT8], dims, [200] * 3, B, lens, np.int32)
    out_ty = O.FP16 if out_dtype == "float16" else O.FP32
    want = oracle_lookup(c, O.SUM, out_ty)
    d = torch.device("cuda")
    t_ = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(d)
    rows_per_dest = 5
    parts = [torch.zeros((rows_per_dest, 68), dtype=getattr(torch, out_dtype), device=d) for _ in range(3)]
    ptrs = torch.tensor([p.data_ptr() for p in parts], dtype=torch.int64, device=d)
    cabi.lookup(t_(c.dev_weights), t_(c.weights_offsets), t_(c.weights_tys), t_(c.D_offsets), 68, 32, t_(c.indices),
                t_(c.offsets), O.SUM, parts[0], dest_outputs=ptrs, rows_per_dest=rows_per_dest, output_stride=68)
    got = torch.cat(parts, 0)[:B].float().cpu().numpy()
    assert_close(got, want, out_ty, "misaligned scatter")

@pytest.mark.parametrize("index_dtype", [np.int32, np.int64])
@pytest.mark.parametrize("weighted", [False, True])
def test_one_wave_launch_with_ragged_bags(index_dtype, weighted):
    """A launch that fills the GPU about once (12 000 bags, 400 000 rows: every warp takes a handful of bags) with bags
    as unequal as they get: empty bags at the very start and end and in long stretches, one bag of 5000 rows, stretches
    of one-row bags, three table types and widths."""
    rng = np.random.default_rng(seed_of("one-wave", index_dtype.__name__, weighted))
    T, B = 3, 4000
    lens = rng.poisson(33, T * B).astype(np.int64)
    lens[:200] = 0
    lens[-300:] = 0
    lens[5000:5600] = 0
    lens[2000:2600] = 1
    lens[7000] = 5000
    lens[7001:7040] = 0
    lens[9000:9010] = 700
    c = make_case(rng, [O.INT8, O.INT4, O.FP16], [128, 64, 32], [5000, 3000, 2000], B, lens, index_dtype, weighted, prune_frac=0.01)
    assert c.indices.size > 350_000
    for pooling, out_ty in ((O.SUM, O.FP16), (O.MEAN, O.FP32)):
        run(c, pooling, out_ty, f"one wave, ragged bags, {index_dtype.__name__}")



@pytest.mark.parametrize("weights_ty", [O.INT8, O.INT4, O.FP16, O.FP8, O.FP32])
@pytest.mark.parametrize("D", [64, 128, 256, 512])
@pytest.mark.parametrize("weighted", [False, True])
def test_bags_that_straddle_lane_group_ranges(weights_ty, D, weighted):
    """Few, very unequal bags per table: one bag of a thousand rows next to empty and tiny ones, so that a
    bag is summed in pieces by several lane groups and put together by its owner; also a table whose bags
    are all empty and a batch of a single bag."""
    rng = np.random.default_rng(seed_of(weights_ty, D, weighted))
    for B, lens in ((5, [0, 1000, 0, 3, 1, 0, 0, 0, 0, 0, 2, 0, 0, 777, 1]), (1, [613, 0, 5]), (3, [1, 1, 1, 0, 0, 0, 64, 64, 65])):
        c = make_case(rng, [weights_ty] * 3, [D] * 3, [300, 50, 1000], B, np.asarray(lens), np.int64, weighted, prune_frac=0.01)
        for pooling, out_ty in ((O.SUM, O.FP16), (O.MEAN, O.FP32)):
            run(c, pooling, out_ty, f"straddle B={B}")


# ---- bags summed in steps of eight rows: edges of the unit widths, precision, operands that are not finite -----------------

def _pool_64(c, pooling):
    """The lookup in float64 and, for every output element, the sum of the magnitudes that went into it."""
    out, mag = np.zeros((c.B, c.total_D)), np.zeros((c.B, c.total_D))
    for t in range(c.T):
        E, D, ty = c.rows[t], c.dims[t], c.tys[t]
        rb = O.row_bytes(ty, D, c.row_alignment)
        rows = c.dev_weights[c.weights_offsets[t]:c.weights_offsets[t] + E * rb].reshape(E, rb)
        scale, bias = np.ones((E, 1)), np.zeros((E, 1))
        if ty in (O.INT8, O.INT4):
            head = rows[:, :4].copy().view(np.float16).astype(np.float64)
            scale, bias = head[:, :1], head[:, 1:]
            codes = rows[:, 4:4 + D] if ty == O.INT8 else np.stack([rows[:, 4:4 + D // 2] & 15, rows[:, 4:4 + D // 2] >> 4], 2).reshape(E, D)
        elif ty in (O.FP16, O.FP32):
            dt = np.dtype(np.float16 if ty == O.FP16 else np.float32)
            codes = rows[:, :dt.itemsize * D].copy().view(dt)
        else:
            b = rows[:, :D].astype(np.int64)
            e, m = (b >> 3) & 15, (b & 7) / 8.0
            codes = np.where(b >> 7, -1.0, 1.0) * np.where(e > 0, (1.0 + m) * 2.0 ** (e - 7.0), m * 2.0 ** -6)
        part = codes.astype(np.float64) * scale
        do = slice(c.D_offsets[t], c.D_offsets[t + 1])
        for b in range(c.B):
            lo, hi = int(c.offsets[t * c.B + b]), int(c.offsets[t * c.B + b + 1])
            i, w = c.indices[lo:hi].astype(np.int64), np.ones(hi - lo) if c.weights is None else c.weights[lo:hi].astype(np.float64)
            i, w = i[i >= 0], w[i >= 0][:, None]
            mul = 1.0 / (hi - lo) if pooling == O.MEAN and hi > lo else 1.0
            out[b, do] = (w * (part[i] + bias[i])).sum(0) * mul
            mag[b, do] = (np.abs(w) * (np.abs(part[i]) + np.abs(bias[i]))).sum(0) * mul
    return out, mag


@pytest.mark.parametrize("weights_ty,dims", [
    (O.INT8, [4, 28, 32, 36, 60, 64]), (O.INT8, [68, 124, 128, 132]), (O.INT8, [252, 256, 260, 516]),
    (O.INT4, [8, 56, 64, 72, 120, 128]), (O.INT4, [136, 248, 256, 264, 520]),
    (O.FP8, [4, 32, 36, 64, 68]), (O.FP8, [128, 132, 256, 260]),
    (O.FP16, [4, 12, 16, 32, 36]), (O.FP16, [64, 68, 128, 132, 260]), (O.FP32, [4, 16, 32, 36, 48, 64]), (O.FP32, [68, 80, 128, 132, 260])])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("out_ty", [O.FP32, O.FP16, O.BF16])
def test_row_widths_at_the_edges_of_the_units(weights_ty, dims, weighted, out_ty):
    """Widths around the unit sizes of pool_run_steps (a row that ends in, at and just past a unit; one and several passes),
    bags of 0 to 9 rows and a long one (step boundaries in every position), pruned rows.  Against float64: every
    term enters with a relative error of at most 2^-22 and every addition rounds to 2^-23 of a partial sum that is
    bounded by the sum of magnitudes, and at most one addition per row is made."""
    rng = np.random.default_rng(seed_of(weights_ty, dims, weighted))
    T, B = len(dims), 21
    lens = rng.integers(0, 10, T * B)
    lens[3] = 67
    c = make_case(rng, [weights_ty] * T, dims, [50] * T, B, lens, np.int64 if weighted else np.int32, weighted, prune_frac=0.03)
    for pooling in (O.SUM, O.MEAN):
        want, mag = _pool_64(c, pooling)
        got = gpu_lookup(c, pooling, out_ty).astype(np.float64)
        rows = np.repeat((c.offsets[1:] - c.offsets[:-1]).reshape(T, B).T, dims, axis=1)
        half_ulp = {O.FP32: 0.0, O.FP16: 2.0 ** -11, O.BF16: 2.0 ** -8}[out_ty]
        bound = mag * (2.0 ** -22 + rows * 2.0 ** -23) + np.abs(want) * half_ulp * 1.01 + (2.0 ** -25 if out_ty == O.FP16 else 1e-38)
        assert np.all(np.abs(got - want) <= bound), f"max excess {(np.abs(got - want) - bound).max()}"


@pytest.mark.parametrize("weights_ty", [O.INT8, O.INT4, O.FP8])
@pytest.mark.parametrize("magnitude", [1e-30, 1e-12, 1.0, 1e12, 1e25, 1e37])
def test_weights_of_any_magnitude(weights_ty, magnitude):
    """Per-sample weights far from one, next to bags of ordinary ones: relative to the magnitudes that go in, the result
    is as good as with weights around one.  (The largest sums of magnitudes here are about 1e38.)"""
    rng = np.random.default_rng(17)
    c = make_case(rng, [weights_ty] * 2, [64, 264], [80, 90], 9, rng.integers(0, 40, 18), np.int64, True)
    c.weights[: int(c.offsets[7])] *= np.float32(magnitude)
    want, mag = _pool_64(c, O.SUM)
    got = gpu_lookup(c, O.SUM, O.FP32).astype(np.float64)
    assert np.all(np.abs(got - want) <= mag * 2.0 ** -17 + 1e-38)      # 40 rows: 2^-22 + 40 * 2^-23


@pytest.mark.parametrize("weights_ty,weighted", [(O.FP16, False), (O.INT8, False), (O.INT8, True), (O.INT4, True)])
def test_infinities_and_nans_stay_in_their_bag(weights_ty, weighted):
    """A row with infinities or NaNs (FP16 payload; INT8 / INT4 bias) changes its own bag only."""
    rng = np.random.default_rng(23)
    c = make_case(rng, [weights_ty] * 2, [128, 36 if weights_ty != O.INT4 else 40], [60, 60], 16, rng.integers(1, 9, 32), np.int32, weighted)
    c.indices[c.indices >= 50] = 1                      # rows 50 .. 53 are used by one bag each
    clean = oracle_lookup(c, O.SUM, O.FP16)
    hit, odd = [0, 5, 18, 31], [np.inf, -np.inf, np.nan, np.inf]
    rb = [O.row_bytes(weights_ty, d, 16) for d in c.dims]
    for k, (bag, value) in enumerate(zip(hit, odd)):
        t = bag // 16
        c.indices[int(c.offsets[bag])] = 50 + k
        at = int(c.weights_offsets[t]) + (50 + k) * rb[t] + (2 * 7 if weights_ty == O.FP16 else 2)
        c.dev_weights[at:at + 2] = np.frombuffer(np.float16(value).tobytes(), dtype=np.uint8)
    got = gpu_lookup(c, O.SUM, O.FP16)
    want = oracle_lookup(c, O.SUM, O.FP16)
    for t in range(2):
        cols = slice(c.D_offsets[t], c.D_offsets[t + 1])
        touched = np.zeros(16, bool)
        touched[[b - 16 * t for b in hit if b // 16 == t]] = True
        assert np.allclose(got[~touched][:, cols], clean[~touched][:, cols], rtol=1e-3, atol=1e-3)
        assert np.array_equal(np.isnan(got[touched][:, cols]), np.isnan(want[touched][:, cols]))
        assert np.allclose(got[touched][:, cols], want[touched][:, cols], rtol=1e-3, atol=1e-3, equal_nan=True)


@pytest.mark.parametrize("weights_ty,dims", [(O.INT8, [4, 12, 8, 40]), (O.INT4, [8, 40, 24, 136]), (O.FP16, [8, 20, 2, 40]), (O.FP8, [4, 24, 8, 100]),
                                             (O.FP32, [3, 4, 20, 8])])
@pytest.mark.parametrize("out_ty", [O.FP32, O.FP16, O.BF16])
def test_sequence_rows_of_any_width(weights_ty, dims, out_ty):
    """Sequence mode with tables of several widths (the narrower ones zero-filled), widths that are not whole 16-byte pieces of
    the output, output rows that are not 16-byte aligned, pruned rows, and counts around the 64 positions of a warp."""
    rng = np.random.default_rng(seed_of("sequence", weights_ty, dims))
    lens = np.array([0, 63, 64, 65, 1, 0, 130, 5])
    for ds in (dims, dims[:2]):
        c = make_case(rng, [weights_ty] * len(ds), ds, [70] * len(ds), 2, lens[:2 * len(ds)], np.int64, False, prune_frac=0.05)
        run(c, O.NONE, out_ty, f"sequence dims={ds}")


@pytest.mark.parametrize("fp8", [(5, 15), (3, 3), (2, 1), (7, 63)])
@pytest.mark.parametrize("weighted", [False, True])
def test_fp8_formats(fp8, weighted):
    """FP8 rows of other exponent widths and biases, in streams (64, 128, 256) and in steps of eight rows (36, 260)."""
    rng = np.random.default_rng(seed_of("fp8", fp8, weighted))
    c = make_case(rng, [O.FP8] * 5, [64, 36, 128, 260, 256], [60] * 5, 7, rng.integers(0, 30, 35), np.int32, weighted, prune_frac=0.03)
    run(c, O.SUM, O.FP32, f"fp8={fp8}", fp8=fp8)
    run(c, O.MEAN, O.FP16, f"fp8={fp8}", fp8=fp8)


def _one_table_of_rows(ty, D, headers, codes, idx, offsets, B, weights=None):
    """A table whose row r has the fp16 pair headers[r] and the codes codes[r]."""
    rb = O.row_bytes(ty, D, 16)
    rows = np.zeros((len(headers), rb), np.uint8)
    for r, (scale, bias) in enumerate(headers):
        rows[r, :4] = np.frombuffer(np.array([scale, bias], np.float16).tobytes(), np.uint8)
        q = np.asarray(codes[r], np.uint8)
        rows[r, 4:4 + (D if ty == O.INT8 else D // 2)] = q if ty == O.INT8 else q[0::2] | (q[1::2] << 4)
    dev, wo, wt, do = O.concat_tables([rows], [ty], [D])
    return Case(dev, wo, wt, do, np.asarray(idx, np.int32), np.asarray(offsets, np.int32), weights, [ty], [D], [len(headers)], B)


@pytest.mark.parametrize("weights_ty", [O.INT8, O.INT4])
@pytest.mark.parametrize("D", [64, 128, 256, 512])
@pytest.mark.parametrize("weighted", [False, True])
def test_pieces_of_a_bag_are_added_without_their_cancelled_parts(weights_ty, D, weighted):
    """A bag of 64 rows that several lane groups sum: 32 rows of code * 2^-10, then 32 rows of code * scale - 32768 = 0 with
    code * scale = 32768.  Every lane group has rows of one kind only (2, 4 or 8 equal ranges), every sum is a multiple of
    2^-10 below 2^13 or of 2^15 below 2^21, so nothing rounds as long as the pieces are handed over with their
    biases: the result is exact.  With the codes' sums added first, 2^20 would take the bits below 2^-3 away."""
    small = np.arange(D) % (255 if weights_ty == O.INT8 else 15) + 1
    big = 64 if weights_ty == O.INT8 else 8
    c = _one_table_of_rows(weights_ty, D, [(2.0 ** -10, 0.0), (32768.0 / big, -32768.0)], [small, np.full(D, big)],
                           [0] * 32 + [1] * 32, [0, 64], 1, np.ones(64, np.float32) if weighted else None)
    assert np.array_equal(gpu_lookup(c, O.SUM, O.FP32)[0], (small * 2.0 ** -5).astype(np.float32))


@pytest.mark.parametrize("weights_ty", [O.INT8, O.INT4])
@pytest.mark.parametrize("D", [40, 128, 520])
@pytest.mark.parametrize("weighted", [False, True])
def test_mean_of_rows_that_cancel_is_zero(weights_ty, D, weighted):
    """Rows of code * scale - 32768 = 0: the codes' sum and the biases' sum are whole multiples of 2^15 and cancel exactly, so
    their mean over 3, 5 or 7 rows is exactly zero; a bias that is divided (and rounded) by itself leaves a remainder.  9000
    bags: a warp takes several in a row, whole ones and such that lane groups share."""
    big = 64 if weights_ty == O.INT8 else 8
    offsets = np.cumsum([0] + [3, 5, 7] * 3000)
    c = _one_table_of_rows(weights_ty, D, [(32768.0 / big, -32768.0)], [np.full(D, big)], [0] * int(offsets[-1]), offsets, 9000,
                           np.ones(int(offsets[-1]), np.float32) if weighted else None)
    assert np.all(gpu_lookup(c, O.MEAN, O.FP32) == 0.0)


@pytest.mark.parametrize("weights_ty", [O.INT8, O.FP16])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("dims", [[20, 128, 528], [64, 128, 256], [20, 36, 1]])
def test_bad_offsets_inside_a_run_are_reported_bag_by_bag(weights_ty, weighted, dims):
    """Offsets that go backwards, past the end of `indices` or below zero between good ones (8000 bags per table: a warp takes
    eleven in a row): bit 8, the bags they bound come out as zeros, and every other bag as if nothing had happened."""
    import torch
    from fbgemm_ascend_b200 import cabi

    rng = np.random.default_rng(seed_of("bad offsets", weights_ty, weighted, dims))
    T, B = 3, 8000
    c = make_case(rng, [weights_ty] * T, dims, [100] * T, B, rng.integers(0, 5, T * B), np.int64, weighted)
    n = c.indices.size
    for t in range(T):
        for b, value in ((4, 10 ** 9), (1003, -7), (4007, None), (6000, n + 1)):
            i = t * B + b
            c.offsets[i] = c.offsets[i - 1] - 3 if value is None else value
    start, end = c.offsets[:-1], c.offsets[1:]
    sane = (start >= 0) & (end >= start) & (end <= n)
    assert int((~sane).sum()) == 7 * T
    # the good bags, one after the other (the one behind a backward step has its neighbour's last three rows as well)
    pieces = [slice(int(s), int(e)) if ok else slice(0, 0) for s, e, ok in zip(start, end, sane)]
    idx = np.concatenate([c.indices[p] for p in pieces])
    offsets = np.concatenate([[0], np.cumsum([p.stop - p.start for p in pieces])]).astype(np.int64)
    good = Case(c.dev_weights, c.weights_offsets, c.weights_tys, c.D_offsets, idx, offsets,
                None if c.weights is None else np.concatenate([c.weights[p] for p in pieces]), c.tys, c.dims, c.rows, B)
    d = torch.device("cuda")
    t_ = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(d)
    flag = torch.zeros(1, dtype=torch.int32, device=d)
    out = torch.full((B, c.total_D), 7.0, dtype=torch.float32, device=d)
    cabi.lookup(t_(c.dev_weights), t_(c.weights_offsets), t_(c.weights_tys), t_(c.D_offsets), c.total_D, max(dims), t_(c.indices),
                t_(c.offsets), O.SUM, out, indice_weights=None if c.weights is None else t_(c.weights), error_flag=flag)
    assert int(flag.item()) == 8
    got, want = out.cpu().numpy(), _pool_64(good, O.SUM)
    assert np.all(np.abs(got - want[0]) <= want[1] * (2.0 ** -22 + 2.0 ** -23 * np.diff(offsets).reshape(T, B).T.repeat(dims, axis=1)) + 1e-38)
    for t in range(T):
        bad = ~sane[t * B:(t + 1) * B]
        assert np.all(got[bad][:, c.D_offsets[t]:c.D_offsets[t + 1]] == 0.0)


@pytest.mark.parametrize("weights_ty", [O.INT8, O.INT4, O.FP16, O.FP8, O.FP32])
@pytest.mark.parametrize("dims", [[16, 20], [16, 18], [16, 17], [128, 132], [136, 140]])
@pytest.mark.parametrize("out_ty", [O.FP32, O.FP16, O.BF16])
def test_sequence_rows_that_are_not_whole_pieces(weights_ty, dims, out_ty):
    """Output rows that start on 8, 4 or 2 bytes (widths of an even table set by an odd one beside it)."""
    rng = np.random.default_rng(seed_of("sequence rows", weights_ty, dims))
    c = make_case(rng, [weights_ty] * 2, dims, [70] * 2, 3, np.array([40, 64, 3, 9, 0, 70]), np.int64, False, prune_frac=0.05)
    run(c, O.NONE, out_ty, f"sequence dims={dims}")
