"""Parity of sum / mean / max / min and sum_to_shape against the CPU oracle, through the
C ABI, on a B200.

Bar: integers bit-exact (wrapping sums are order-independent); max / min bit-exact for
every dtype (the result is one of the inputs); float sums and means against the oracle's
wide-accumulator evaluation of the same formulas: f32 within 1e-4, f64 1e-12, bf16 / f16
2e-2, each relative to max(|ref|, sqrt(R) * sigma) where R is the number of folded terms
(the natural scale of a sum of R zero-mean terms).  Output buffers are handed over dirty
(the ops must overwrite), and every case is run twice to check bitwise determinism.
Shapes are chosen to hit every kernel: thread / warp / block rows, split rows, vector and
scalar column strips, split columns, the [O,R,I] middle fold, and the literal scatter
path (several reduced dims, non-contiguous input, broadcast input, partial factors).
"""
import numpy as np
import pytest

import harness as H
from maidenx_b200 import dtypes as D

pytestmark = pytest.mark.gpu

SUM_TOL = {"f32": 1e-4, "f64": 1e-12, "bf16": 2e-2, "f16": 2e-2}


def dim_cases():
    """(name, dims, strides or None for contiguous, reduced dims, offset)"""
    return [
        ("rows-thread", [300, 7], None, [1], 0),
        ("rows-warp", [2000, 96], None, [1], 0),
        ("rows-warp-odd", [777, 101], None, [1], 0),
        ("rows-block", [40, 5000], None, [1], 0),
        ("rows-block-vec", [24, 4096], None, [1], 0),
        ("rows-split", [3, 70001], None, [1], 0),
        ("sum-all", [123457], None, [0], 0),
        ("cols-vec", [500, 256], None, [0], 0),
        ("cols-odd", [333, 77], None, [0], 0),
        ("cols-split", [4000, 64], None, [0], 0),
        ("cols-narrow", [900, 3], None, [0], 0),
        ("middle", [6, 50, 40], None, [1], 0),
        ("middle-narrow", [5, 33, 2], None, [1], 0),
        ("offset1", [64, 33], None, [0], 1),
        ("offset1-rows", [33, 64], None, [1], 1),
        ("len1", [17, 1, 9], None, [1], 0),
        ("two-dims", [6, 7, 8], None, [0, 2], 0),
        ("transposed-input", [12, 10], [1, 12], [0], 0),
        ("broadcast-input", [4, 6], [0, 1], [0], 0),
    ]


def _run_dim(be, op, dt, dims, strides, red, off, store):
    st = strides or H.contiguous_strides(dims)
    return H.run_reduce(be, op, dt, dims, st, [dims[d] for d in red], [st[d] for d in red], off, store)


def _buffer_len(dims, strides, off):
    if strides is None:
        return H.numel(dims) + off
    return sum((d - 1) * s for d, s in zip(dims, strides)) + 1 + off


@pytest.mark.parametrize("op", ["sum", "mean", "max", "min"])
def test_dim_reductions(oracle, cuda, op):
    from oracle import binding
    rng = np.random.default_rng({"sum": 1, "mean": 2, "max": 3, "min": 4}[op])
    for dt in (D.FLOATS if op == "mean" else D.ARITH):
        for name, dims, strides, red, off in dim_cases():
            blen = _buffer_len(dims, strides, off)
            if op in ("max", "min"):
                store = H.full_range_store(rng, dt, blen)
            elif dt.kind == "float":
                store = H.random_store(rng, dt, blen, dist="normal")
            else:
                store = H.full_range_store(rng, dt, blen)  # wrapping sums
            binding.set_wide(op in ("sum", "mean") and dt.kind == "float")
            try:
                ref = _run_dim(oracle, op, dt, dims, strides, red, off, store)
            finally:
                binding.set_wide(False)
            got = _run_dim(cuda, op, dt, dims, strides, red, off, store)
            again = _run_dim(cuda, op, dt, dims, strides, red, off, store)
            assert got.tobytes() == again.tobytes() or (dt.kind == "float" and name in ("two-dims", "transposed-input", "broadcast-input")), \
                f"{name} {op}_{dt.name}: not deterministic"
            if op in ("max", "min") or dt.kind != "float":
                H.assert_same(op, dt, got, ref, what=name)
            else:
                folded = 1
                for d in red:
                    folded *= dims[d]
                scale = np.sqrt(folded) * (1.0 if op == "sum" else 1.0 / folded)
                H.assert_same(op, dt, got, ref, float_rel=SUM_TOL[dt.name], what=name, scale=scale)


def shape_cases():
    """(name, in_dims, strides or None, out_dims, offset)"""
    return [
        ("lead-fold", [64, 96], None, [1, 96], 0),                 # [R, K]
        ("lead-fold-3d", [8, 16, 40], None, [1, 1, 40], 0),        # merged [R, K]
        ("trail-fold", [50, 333], None, [50, 1], 0),               # [K, R]
        ("full-fold", [9, 11, 13], None, [1, 1, 1], 0),            # [R]
        ("middle-fold", [7, 30, 24], None, [7, 1, 24], 0),         # [K, R, K]
        ("bias-fold", [4, 6, 5, 5], None, [1, 6, 1, 1], 0),        # [R, K, R]: literal scatter
        ("no-fold", [5, 8], None, [5, 8], 1),
        ("partial", [4, 6], None, [2, 3], 0),                      # block fold by 2 x 2
        ("offset1", [2, 3], None, [1, 3], 1),
        ("transposed-input", [6, 4], [1, 6], [1, 4], 0),
    ]


def test_sum_to_shape(oracle, cuda):
    from oracle import binding
    rng = np.random.default_rng(11)
    for dt in D.ARITH:
        for name, dims, strides, odims, off in shape_cases():
            blen = _buffer_len(dims, strides, off)
            store = H.random_store(rng, dt, blen, dist="normal") if dt.kind == "float" else H.full_range_store(rng, dt, blen)
            st = strides or H.contiguous_strides(dims)
            binding.set_wide(dt.kind == "float")
            try:
                ref = H.run_sum_to_shape(oracle, dt, dims, st, odims, off, store)
            finally:
                binding.set_wide(False)
            got = H.run_sum_to_shape(cuda, dt, dims, st, odims, off, store)
            if dt.kind != "float":
                H.assert_same("sum_to_shape", dt, got, ref, what=name)
            else:
                folded = H.numel(dims) // H.numel(odims)
                H.assert_same("sum_to_shape", dt, got, ref, float_rel=SUM_TOL[dt.name], what=name, scale=np.sqrt(folded))


def test_f32_max_of_only_negative_infinity_is_type_min(oracle, cuda):
    """max starts from f32::MIN, not -inf (crates/maidenx_cpu/src/ops/reduction.rs:605), and NaNs never win."""
    x = np.array([-np.inf, np.nan, -np.inf, -np.inf, np.nan, -np.inf], dtype=np.float32)
    ref = H.run_reduce(oracle, "max", D.F32, [2, 3], [3, 1], [3], [1], 0, x)
    got = H.run_reduce(cuda, "max", D.F32, [2, 3], [3, 1], [3], [1], 0, x)
    assert np.array_equal(ref, got) and got[0] == np.finfo(np.float32).min


@pytest.mark.parametrize("shape", [(2, 3, 5), (3, 300, 49), (256, 64, 49), (64, 7, 9), (130, 33, 1), (4, 8, 4096), (5, 3, 1027), (2, 2, 70001), (700, 2, 3)], ids=str)
def test_outer_and_inner_dims_folded_around_a_kept_one(oracle, cuda, shape):
    """sum_to_shape [Q, O, I] -> [1, O, 1], the gradient of a per-channel operand: both orders of the two passes, split and
    unsplit, vector and scalar strips.  Bound: the sums' tolerance of this file (f32 and wider accumulation, one rounding)."""
    from oracle import binding
    q, o, i = shape
    rng = np.random.default_rng(q * 1000 + o)
    for dt in (D.F32, D.BF16, D.F16, D.F64, D.I32, D.U8):
        dims, out_dims = [q, o, i], [1, o, 1]
        x = H.random_store(rng, dt, H.numel(dims) + 1, dist="normal") if dt.kind == "float" else H.full_range_store(rng, dt, H.numel(dims) + 1)
        for off in (0, 1):
            binding.set_wide(True)
            try:
                ref = H.run_sum_to_shape(oracle, dt, dims, H.contiguous_strides(dims), out_dims, off, x)
            finally:
                binding.set_wide(False)
            got = H.run_sum_to_shape(cuda, dt, dims, H.contiguous_strides(dims), out_dims, off, x)
            again = H.run_sum_to_shape(cuda, dt, dims, H.contiguous_strides(dims), out_dims, off, x)
            assert np.array_equal(got, again)
            H.assert_same("sum_to_shape", dt, got, ref, float_rel=SUM_TOL.get(dt.name, 0.0), what=str((shape, off)), scale=np.sqrt(q * i))


@pytest.mark.parametrize("dt", [D.F32, D.BF16, D.I32, D.U8, D.F64], ids=lambda d: d.name)
@pytest.mark.parametrize("shape", [(303200, 8), (151600, 56), (76000, 13), (38000, 100), (37900, 30), (700, 31), (700, 33), (700, 1023), (700, 1032), (151700, 16), (9000, 24),
                                   (700, 128), (700, 129), (700, 255), (700, 2047)], ids=str)
def test_rows_shared_by_part_of_a_warp(oracle, cuda, shape, dt):
    """Row lengths around the lanes a row gets (one thread, 4 to 32 lanes, then a warp that walks the row in trips of four or two loads), and row counts on both sides of the
    form with four rows per group; the sum within this file's tolerance, the maximum exact."""
    from oracle import binding
    rows, r = shape
    rng = np.random.default_rng(rows + r)
    x = H.random_store(rng, dt, rows * r, dist="normal") if dt.kind == "float" else H.full_range_store(rng, dt, rows * r)
    for op in ("sum", "max"):
        binding.set_wide(True)
        try:
            ref = _run_dim(oracle, op, dt, [rows, r], None, [1], 0, x)
        finally:
            binding.set_wide(False)
        got = _run_dim(cuda, op, dt, [rows, r], None, [1], 0, x)
        H.assert_same(op, dt, got, ref, float_rel=SUM_TOL.get(dt.name, 0.0) if op == "sum" else 0.0, what=str((op, shape)), scale=np.sqrt(r))


@pytest.mark.parametrize("shape", [(2, 40000, 5), (2, 40000, 7), (3, 33000, 4), (2, 40000, 60), (5, 700000, 2), (3, 30001, 200)], ids=str)
def test_outer_folds_of_many_outputs(oracle, cuda, shape):
    """Both sides of the line between the scatter and the two passes (many outputs of few elements), and partial results beyond the
    thread's scratch block.  Integers exact; sums of ones of a range that every type holds, so floats are exact too."""
    q, o, i = shape
    rng = np.random.default_rng(q * 1000 + o)
    for dt in (D.F32, D.BF16, D.F64, D.I64, D.U8):
        n = q * o * i
        x = D.encode(rng.integers(0, 2, n).astype(np.float32 if dt is not D.F64 else np.float64), dt) if dt.kind == "float" else rng.integers(0, 2, n).astype(dt.np_storage)
        got = D.decode(H.run_sum_to_shape(cuda, dt, [q, o, i], H.contiguous_strides([q, o, i]), [1, o, 1], 0, x), dt)
        want = np.asarray(D.decode(x, dt)).reshape(q, o, i).sum(axis=(0, 2), dtype=np.float64)
        tol = 2.0 ** -8 if dt.name == "bf16" else 0.0          # one rounding of the sum; 256 and more have no exact bf16
        if dt.name == "u8":
            want %= 256
        assert np.all(np.abs(np.asarray(got, dtype=np.float64) - want) <= tol * want), dt.name


@pytest.mark.parametrize("dt", [D.F32, D.BF16, D.F16, D.U8, D.I16, D.I32], ids=lambda d: d.name)
def test_ragged_rows_by_the_words_they_lie_in(oracle, cuda, dt):
    """Rows that are no whole aligned vectors, from an aligned base and from every place inside a word: the first and last word of a row belong to its
    neighbours too, whose elements (the largest and smallest values) must not count."""
    from oracle import binding
    rng = np.random.default_rng(dt.size)
    vec = 16 // dt.size
    for r in (8 * vec + 1, 9 * vec - 1, 15 * vec + 1, 17 * vec + 2, 31 * vec + 1, 32 * vec + 1, 33 * vec - 1, 2047):
        o = 701
        for off in (0, 1, vec - 1):
            x = H.random_store(rng, dt, o * r + off, dist="normal") if dt.kind == "float" else H.random_store(rng, dt, o * r + off)
            for op in ("sum", "mean", "max"):
                if op == "mean" and dt.kind != "float":
                    continue
                binding.set_wide(dt.kind == "float" and op != "max")
                try:
                    ref = H.run_reduce(oracle, op, dt, [o, r], [r, 1], [r], [1], off, x)
                finally:
                    binding.set_wide(False)
                got = H.run_reduce(cuda, op, dt, [o, r], [r, 1], [r], [1], off, x)
                H.assert_same(op, dt, got, ref, float_rel=SUM_TOL.get(dt.name, 0.0) if op != "max" else 0.0, what=str((op, r, off)), scale=np.sqrt(r) if op == "sum" else 1.0)


@pytest.mark.parametrize("dt", [D.F32, D.BF16, D.U8, D.I32], ids=lambda d: d.name)
def test_ragged_rows_on_both_sides_of_the_rules_lines(oracle, cuda, dt):
    """Rows of up to 16, up to 32 and more words, in counts on both sides of where a group of lanes takes four rows at a time (256 and 1024 rows an SM); a last
    group that is not full."""
    from oracle import binding
    rng = np.random.default_rng(dt.size + 5)
    vec = 16 // dt.size
    rows = {4: (37887, 37889), 2: (37889, 151551, 151555), 1: (37889,)}[dt.size]
    for r in (8 * vec + 1, 14 * vec + 3, 15 * vec + 3, 30 * vec + 1, 31 * vec + 3):
        for o in rows:
            x = H.random_store(rng, dt, o * r + 1, dist="normal") if dt.kind == "float" else H.random_store(rng, dt, o * r + 1)
            for op in ("sum", "max"):
                binding.set_wide(dt.kind == "float" and op != "max")
                try:
                    ref = H.run_reduce(oracle, op, dt, [o, r], [r, 1], [r], [1], 1, x)
                finally:
                    binding.set_wide(False)
                got = H.run_reduce(cuda, op, dt, [o, r], [r, 1], [r], [1], 1, x)
                H.assert_same(op, dt, got, ref, float_rel=SUM_TOL.get(dt.name, 0.0) if op != "max" else 0.0, what=str((op, r, o)), scale=np.sqrt(r) if op == "sum" else 1.0)


@pytest.mark.parametrize("dt", [D.F32, D.BF16, D.F64, D.I32, D.U8, D.U64], ids=lambda d: d.name)
@pytest.mark.parametrize("shape", [(769, 33), (1600, 1), (17683, 43), (9999, 100), (20011, 129), (3, 5000, 31), (6500, 132), (40000, 2)], ids=str)
def test_columns_cut_into_many_parts(oracle, cuda, shape, dt):
    """The last block of a strip folds its parts with several threads a column: on both sides of the number of parts from which on, strips with columns missing, fewer parts than threads
    would share, several outer indices; twice, with the same bits (float sums: the file's bounds)."""
    rng = np.random.default_rng(sum(shape))
    a = H.random_store(rng, dt, int(np.prod(shape)), dist="normal") if dt.kind == "float" else H.random_store(rng, dt, int(np.prod(shape)))
    dim = len(shape) - 2
    from oracle import binding
    for op in ("sum", "max", "min") + (("mean",) if dt.kind == "float" else ()):
        got = _run_dim(cuda, op, dt, list(shape), None, [dim], 0, a)
        binding.set_wide(True)
        try:
            ref = _run_dim(oracle, op, dt, list(shape), None, [dim], 0, a)
        finally:
            binding.set_wide(False)
        exact = dt.kind != "float" or op in ("max", "min")
        if exact:
            assert np.array_equal(got, ref), op
        else:
            scale = np.sqrt(shape[dim]) / (shape[dim] if op == "mean" else 1.0)
            H.assert_same(op, dt, got, ref, float_rel=SUM_TOL[dt.name], scale=scale, what=f"{op} {shape}")
        assert np.array_equal(got, _run_dim(cuda, op, dt, list(shape), None, [dim], 0, a)), op
