"""Parity of matmul / matmul_backward against the CPU oracle, through the C ABI, on a B200.

Bar: integers bit-exact (wrapping); f32 / f64 bit-exact against the oracle's faithful mode
(element-type accumulation, k ascending — the SIMT kernel keeps that order and does not
contract multiplies and adds); bf16 / f16 against the oracle's wide mode (f32 accumulation,
one rounding): bit-exact on the SIMT path, within rel 2e-2 of max(|ref|, sqrt(K)) where the
tensor-core path (different summation order) takes the call.
Cases include the reference's index quirks: only strides[0] is used for the batch of
rank > 3 operands, rank-1 B is indexed by the output column alone, and terms whose linear
index reaches num_els * k are skipped (crates/maidenx_cpu/src/ops/matmul.rs:55-113).
"""
import zlib

import ctypes

import numpy as np
import pytest

import harness as H
from maidenx_b200 import dtypes as D

pytestmark = pytest.mark.gpu


def zlib_seed(text):
    return zlib.crc32(text.encode())


def fwd_cases():
    """(name, out_shape, a_shape, b_shape, a_strides, b_strides, a_off, b_off, a_len, b_len)"""
    cs = H.contiguous_strides
    out = []

    def add(name, o, a, b, ast=None, bst=None, aoff=0, boff=0, alen=None, blen=None):
        ast = ast or cs(a)
        bst = bst or cs(b)
        alen = alen or (sum((d - 1) * s for d, s in zip(a, ast)) + 1 + aoff)
        blen = blen or (sum((d - 1) * s for d, s in zip(b, bst)) + 1 + boff)
        out.append((name, o, a, b, ast, bst, aoff, boff, alen, blen))

    add("mm-small", [2, 2], [2, 2], [2, 2], aoff=1, boff=1)
    add("mm-odd", [65, 33], [65, 70], [70, 33])
    add("mm-tiles", [128, 192], [128, 96], [96, 192])
    add("mm-tall-k", [7, 5], [7, 1000], [1000, 5])
    add("long-k", [3, 2], [3, 5000], [5000, 2])                            # few outputs, long reduction: one block per output element
    add("long-k-tn", [1, 3], [1, 10000], [10000, 3], ast=[1, 1])           # the weight gradient of the README example
    add("nt-linear", [50, 24], [50, 40], [40, 24], bst=[1, 40])            # x . W^T with W [24, 40]
    add("tn", [30, 20], [30, 16], [16, 20], ast=[1, 30])
    add("batched", [3, 20, 17], [3, 20, 30], [3, 30, 17])
    add("batched-span", [5, 50, 9], [5, 50, 8], [5, 8, 9])                 # 64-row tiles span batches
    add("batch-bcast-b", [4, 10, 6], [4, 10, 7], [4, 7, 6], bst=[0, 6, 1])  # B broadcast over the batch
    add("rank4", [2, 3, 4, 6], [2, 3, 4, 5], [2, 3, 5, 6])                 # batch index uses strides[0] only
    add("vec-mat", [1, 9], [1, 12], [12, 9])
    add("mat-vec", [8, 1], [8, 12], [12, 1])
    add("rank1-a", [1, 4], [5], [5, 4])                                    # contiguous formulas, m = 1
    add("rank1-b", [6, 1], [6, 5], [5])                                    # contiguous formulas, n = 1
    add("rank1-a-strided", [3, 4], [5], [5, 4], ast=[2], alen=9)           # literal: A indexed by k only, rows repeat
    add("rank1-b-strided", [6, 4], [6, 5], [4], bst=[2], blen=7)           # literal: B indexed by n only
    add("sliced-a-skips", [6, 1], [6, 4], [4, 1], ast=[16, 1])             # indices >= num_els * k are dropped
    # large enough for the tensor-core path (bf16 / f16): ragged M, N, K tiles; NT and NN operand layouts
    add("tc-nt", [200, 264], [200, 392], [392, 264], bst=[1, 392])
    add("tc-nt-tiles", [384, 512], [384, 256], [256, 512], bst=[1, 256])
    add("tc-nn", [136, 520], [136, 320], [320, 520])
    add("tc-tn", [264, 256], [264, 392], [392, 256], ast=[1, 264])          # A is the transposed view of a [392, 264] matrix
    add("tc-tt", [256, 264], [256, 384], [384, 264], ast=[1, 256], bst=[1, 384])
    # batched products on the tensor cores: dense batches, and one operand shared by every batch (stride 0), which is
    # how a [Cout, K] weight meets a [B, K, P] column buffer (crates/maidenx_tensor/src/ops/matmul.rs:161-225)
    add("tc-batched", [3, 136, 264], [3, 136, 200], [3, 200, 264])
    add("tc-batch-bcast-a", [4, 72, 264], [4, 72, 392], [4, 392, 264], ast=[0, 392, 1], alen=72 * 392)
    add("tc-batch-bcast-b-nt", [3, 200, 264], [3, 200, 392], [3, 392, 264], bst=[0, 1, 392], blen=392 * 264)
    add("tc-batched-tn", [2, 264, 256], [2, 264, 392], [2, 392, 256], ast=[392 * 264, 1, 264])
    return out


def _inputs(rng, dt, n):
    if dt.kind == "float":
        return H.random_store(rng, dt, n, dist="normal")
    return H.full_range_store(rng, dt, n)


@pytest.mark.parametrize("dt", D.ARITH, ids=lambda d: d.name)
def test_matmul_forward(oracle, cuda, dt):
    from oracle import binding
    rng = np.random.default_rng(100 + D.ARITH.index(dt))
    for name, o, a_sh, b_sh, ast, bst, aoff, boff, alen, blen in fwd_cases():
        meta = H.matmul_metadata(o, a_sh, b_sh, ast, bst, aoff, boff)
        a, b = _inputs(rng, dt, alen), _inputs(rng, dt, blen)
        n = H.numel(o)
        # f32 products large enough for the tensor cores run on split tf32 operands: summation order and the
        # last bits differ from element-type accumulation, so they are held to the stated 1e-4 against the wide oracle
        f32_tc = dt.name == "f32" and name.startswith("tc-")
        long_k = name.startswith("long-k") and dt.kind == "float"   # summed in a different order than the element-type loop
        binding.set_wide(dt.name in ("bf16", "f16") or f32_tc or long_k)
        try:
            ref = H.run_matmul(oracle, dt, meta, n, a, b)
        finally:
            binding.set_wide(False)
        got = H.run_matmul(cuda, dt, meta, n, a, b)
        if dt.name in ("bf16", "f16"):
            H.assert_same("matmul", dt, got, ref, float_rel=2e-2, what=name, scale=np.sqrt(a_sh[-1]))
        elif long_k:
            H.assert_same("matmul", dt, got, ref, float_rel=1e-4 if dt.name == "f32" else 1e-12, what=name, scale=10 * np.sqrt(a_sh[-1]))
        elif f32_tc:
            H.assert_same("matmul", dt, got, ref, float_rel=1e-4, what=name, scale=np.sqrt(a_sh[-1]))
            # split tf32 is far inside that bound (a few 1e-6: the tensor core's truncating accumulation over one
            # 128-wide K chunk); a plain tf32 product (error ~5e-4) would not pass this one
            H.assert_same("matmul", dt, got, ref, float_rel=1e-5, what=name + " (split-tf32 accuracy)", scale=np.sqrt(a_sh[-1]))
        else:
            H.assert_same("matmul", dt, got, ref, what=name)


def bwd_cases():
    """(name, out_shape, a_shape, b_shape, a_off, b_off)"""
    return [
        ("mm", [2, 2], [2, 2], [2, 2], 1, 1),
        ("mm-odd", [37, 21], [37, 45], [45, 21], 0, 0),
        ("mm-tiles", [128, 64], [128, 96], [96, 64], 0, 0),
        ("batched", [3, 10, 7], [3, 10, 12], [3, 12, 7], 2, 0),
        ("mat-vec", [9, 1], [9, 14], [14, 1], 0, 3),
        ("vec-mat", [1, 6], [1, 11], [11, 6], 0, 0),
        ("tc", [264, 256], [264, 384], [384, 256], 0, 0),   # tensor-core path for bf16 / f16
    ]


@pytest.mark.parametrize("dt", D.ARITH, ids=lambda d: d.name)
def test_matmul_backward(oracle, cuda, dt):
    from oracle import binding
    rng = np.random.default_rng(200 + D.ARITH.index(dt))
    cs = H.contiguous_strides
    for name, o, a_sh, b_sh, aoff, boff in bwd_cases():
        meta = H.matmul_metadata(o, a_sh, b_sh, cs(a_sh), cs(b_sh), aoff, boff)
        nea, neb = H.numel(a_sh), H.numel(b_sh)
        a, b, g = _inputs(rng, dt, nea + aoff), _inputs(rng, dt, neb + boff), _inputs(rng, dt, H.numel(o))
        for want_a, want_b in ((True, True), (True, False), (False, True)):
            f32_tc = dt.name == "f32" and name == "tc"
            binding.set_wide(dt.name in ("bf16", "f16") or f32_tc)
            try:
                ref = H.run_matmul_backward(oracle, dt, meta, nea, neb, g, a, b, want_a, want_b)
            finally:
                binding.set_wide(False)
            got = H.run_matmul_backward(cuda, dt, meta, nea, neb, g, a, b, want_a, want_b)
            for key in ref:
                if dt.name in ("bf16", "f16") or f32_tc:
                    k = o[-1] if key == "ga" else (o[-2] if len(o) >= 2 else 1)
                    H.assert_same("matmul_backward", dt, got[key], ref[key], float_rel=1e-4 if f32_tc else 2e-2, what=f"{name}/{key}", scale=np.sqrt(k))
                else:
                    H.assert_same("matmul_backward", dt, got[key], ref[key], what=f"{name}/{key}")


def test_matmul_backward_ignores_strides_of_a_transposed_view(oracle, cuda):
    """Linear's backward hands matmul_backward the transposed weight view; both backends read it
    as if it were contiguous (crates/maidenx_cpu/src/ops/matmul.rs:211-217)."""
    dt = D.F32
    rng = np.random.default_rng(5)
    o, a_sh, b_sh = [6, 4], [6, 5], [5, 4]
    meta = H.matmul_metadata(o, a_sh, b_sh, [5, 1], [1, 5], 0, 0)  # B = W^T view, strides [1, 5]
    a, b, g = _inputs(rng, dt, 30), _inputs(rng, dt, 20), _inputs(rng, dt, 24)
    ref = H.run_matmul_backward(oracle, dt, meta, 30, 20, g, a, b)
    got = H.run_matmul_backward(cuda, dt, meta, 30, 20, g, a, b)
    for key in ref:
        H.assert_same("matmul_backward", dt, got[key], ref[key], what=key)


def test_matmul_backward_scalar_grad(oracle, cuda):
    """out_ndim == 0: every gradient row is grad_output[0] times the other operand (matmul.rs:204-207,240-243)."""
    dt = D.F32
    rng = np.random.default_rng(6)
    meta = [0, 1, 1, 7, 7, 1, 1, 0, 0]  # out_ndim 0, a_shape [7], b_shape [7]
    a, b, g = _inputs(rng, dt, 7), _inputs(rng, dt, 7), _inputs(rng, dt, 1)
    ref = H.run_matmul_backward(oracle, dt, meta, 7, 7, g, a, b)
    got = H.run_matmul_backward(cuda, dt, meta, 7, 7, g, a, b)
    for key in ref:
        H.assert_same("matmul_backward", dt, got[key], ref[key], what=key)


# ---------------------------------------------------------------------------------------
# Tensor-core kernel at benchmark scale: more output tiles than SMs (every CTA walks its
# persistent loop several times, both TMEM accumulators change hands), K = 8192 (128
# k-blocks through the 4-stage ring), a ragged last row-group and ragged edge tiles.
# The oracle's matmul is row-independent, so it is run on a sample of rows only.
# ---------------------------------------------------------------------------------------
def _sample_rows(m, count=32):
    edge = [0, 1, 127, 128, 129, m // 2, m - 129, m - 128, m - 2, m - 1]
    rows = sorted({r for r in edge if 0 <= r < m})
    rng = np.random.default_rng(m)
    while len(rows) < count:
        r = int(rng.integers(0, m))
        if r not in rows:
            rows.append(r)
    return np.array(sorted(rows))


BIG_FWD = [
    # name, M, N, K, a_major, b_major  ("k": K contiguous, "mn": M / N contiguous)
    ("nt-512-tiles", 4096, 4096, 8192, "k", "k"),
    ("nn-512-tiles", 4096, 4096, 8192, "k", "mn"),
    ("tn-512-tiles", 4096, 4096, 8192, "mn", "mn"),
    ("nt-ragged-group", 2216, 840, 8192, "k", "k"),      # 18 row-tiles: the last group of 16 holds two; 40-row and 72-column edge tiles
    ("tt-ragged", 2216, 840, 4104, "mn", "k"),           # ragged K block (4104 = 64 * 64 + 8)
    # few tiles, long reduction: K is cut into slices that run as batches, f32 partials summed by a second kernel
    ("splitk-nt", 200, 264, 32768, "k", "k"),
    ("splitk-tn", 264, 256, 65536, "mn", "mn"),          # the shape class of the conv weight gradient
]


@pytest.mark.parametrize("dt", [D.BF16, D.F16, D.F32], ids=lambda d: d.name)
@pytest.mark.parametrize("case", BIG_FWD, ids=lambda c: c[0])
def test_matmul_forward_many_tiles(oracle, cuda, dt, case):
    from oracle import binding
    name, m, n, k, amaj, bmaj = case
    rng = np.random.default_rng(zlib_seed(name + dt.name))
    a = H.random_store(rng, dt, m * k, dist="normal")
    b = H.random_store(rng, dt, k * n, dist="normal")
    ast = [k, 1] if amaj == "k" else [1, m]
    bst = [1, k] if bmaj == "k" else [n, 1]
    meta = H.matmul_metadata([m, n], [m, k], [k, n], ast, bst, 0, 0)
    got = H.run_matmul(cuda, dt, meta, m * n, a, b).reshape(m, n)
    rows = _sample_rows(m)
    a_rows = (a.reshape(m, k)[rows] if amaj == "k" else a.reshape(k, m)[:, rows].T).copy().reshape(-1)
    smeta = H.matmul_metadata([len(rows), n], [len(rows), k], [k, n], [k, 1], bst, 0, 0)
    binding.set_wide(True)
    try:
        ref = H.run_matmul(oracle, dt, smeta, len(rows) * n, a_rows, b).reshape(len(rows), n)
    finally:
        binding.set_wide(False)
    rel = 2e-2 if dt.name in ("bf16", "f16") else 1e-4
    H.assert_same("matmul", dt, got[rows].reshape(-1), ref.reshape(-1), float_rel=rel, what=name, scale=np.sqrt(k))


@pytest.mark.parametrize("dt", [D.BF16, D.F16, D.F32], ids=lambda d: d.name)
def test_matmul_backward_many_tiles(oracle, cuda, dt):
    """grad_a = g . B^T (reduction over n) and grad_b = A^T . g (reduction over m) with more tiles than SMs."""
    from oracle import binding
    m, k, n = 2216, 4096, 840
    rng = np.random.default_rng(zlib_seed("bwd" + dt.name))
    a = H.random_store(rng, dt, m * k, dist="normal")
    b = H.random_store(rng, dt, k * n, dist="normal")
    g = H.random_store(rng, dt, m * n, dist="normal")
    meta = H.matmul_metadata([m, n], [m, k], [k, n], [k, 1], [n, 1], 0, 0)
    got = H.run_matmul_backward(cuda, dt, meta, m * k, k * n, g, a, b)
    ga, gb = got["ga"].reshape(m, k), got["gb"].reshape(k, n)
    rel = 2e-2 if dt.name in ("bf16", "f16") else 1e-4
    binding.set_wide(True)
    try:
        rows = _sample_rows(m)
        smeta = H.matmul_metadata([len(rows), n], [len(rows), k], [k, n], [k, 1], [n, 1], 0, 0)
        ref = H.run_matmul_backward(oracle, dt, smeta, len(rows) * k, k * n, g.reshape(m, n)[rows].copy().reshape(-1),
                                    np.zeros(len(rows) * k, dt.np_storage), b, want_b=False)["ga"]
        H.assert_same("matmul_backward", dt, ga[rows].reshape(-1), ref, float_rel=rel, what="ga", scale=np.sqrt(n))
        cols = _sample_rows(k)
        smeta = H.matmul_metadata([m, n], [m, len(cols)], [len(cols), n], [len(cols), 1], [n, 1], 0, 0)
        ref = H.run_matmul_backward(oracle, dt, smeta, m * len(cols), len(cols) * n, g, a.reshape(m, k)[:, cols].copy().reshape(-1),
                                    np.zeros(len(cols) * n, dt.np_storage), want_a=False)["gb"]
        H.assert_same("matmul_backward", dt, gb[cols].reshape(-1), ref, float_rel=rel, what="gb", scale=np.sqrt(m))
    finally:
        binding.set_wide(False)


def test_stale_device_wait_report_is_surfaced_and_does_not_poison_later_products(oracle, cuda):
    """A tensor-core kernel whose bounded wait ran out leaves a word in device memory.  The ABI's own
    synchronisation points must report it (callers of the reference ABI never call the mx_* status functions),
    and launches made while the word is still there must compute their product normally.  The word is written
    from the host: no wait has to run out on the GPU."""
    import ctypes
    from maidenx_b200 import _lib, device
    from oracle import binding
    lib = _lib.load()
    poke = lib.mx_debug_tc_gemm_poke_status
    poke.argtypes, poke.restype = [ctypes.c_int], ctypes.c_int
    dt = D.BF16
    rng = np.random.default_rng(77)
    m, n, k = 256, 512, 256
    a, b = H.random_store(rng, dt, m * k, dist="normal"), H.random_store(rng, dt, k * n, dist="normal")
    meta = H.matmul_metadata([m, n], [m, k], [k, n], [k, 1], [1, k], 0, 0)
    binding.set_wide(True)
    try:
        ref = H.run_matmul(oracle, dt, meta, m * n, a, b)
    finally:
        binding.set_wide(False)
    assert poke(3) == 0
    bufs = [device.CudaBuffer.from_host(x) for x in (a, b, np.zeros(m * n, dt.np_storage))]
    try:
        device.dispatch("matmul", dt.name, meta, ctypes.c_size_t(m * n), "META", bufs[0].ptr, bufs[1].ptr, bufs[2].ptr)
        out = np.empty(m * n, dt.np_storage)
        rc = lib.cuda_memcpy_d2h(out.ctypes.data, bufs[2].ptr, out.nbytes)
        assert rc != 0, "the copy that follows the product must report the device-side wait"
        assert lib.mx_last_error() == 5 and lib.mx_last_cuda_error() == 3
        lib.mx_clear_error()
        H.assert_same("matmul", dt, out, ref, float_rel=2e-2, what="product launched over a stale report", scale=np.sqrt(k))
        assert lib.cuda_memcpy_d2h(out.ctypes.data, bufs[2].ptr, out.nbytes) == 0  # reported once, then clear
        assert lib.mx_tc_gemm_status() == 0
    finally:
        lib.mx_clear_error()
        for x in bufs:
            x.free()


@pytest.mark.parametrize("dt", [D.BF16, D.F16], ids=lambda d: d.name)
@pytest.mark.parametrize("case", BIG_FWD, ids=lambda c: c[0])
def test_two_cta_kernel_matches_too(oracle, cuda, dt, case):
    """mx_set_gemm_cta_group(2): pairs of CTAs share the B tile (tcgen05.mma.cta_group::2, matmul_tc2.cu).  Same products
    as the default one-CTA kernel, on every many-tile case: odd numbers of row tiles (a pair with an empty half),
    ragged edges, both operand majors, split-K."""
    from maidenx_b200 import _lib
    lib = _lib.load()
    lib.mx_set_gemm_cta_group(2)
    try:
        test_matmul_forward_many_tiles(oracle, cuda, dt, case)
    finally:
        lib.mx_set_gemm_cta_group(1)


@pytest.mark.parametrize("dt", [D.BF16, D.F16], ids=lambda d: d.name)
def test_two_cta_kernel_on_the_small_batched_and_backward_cases(oracle, cuda, dt):
    from maidenx_b200 import _lib
    lib = _lib.load()
    lib.mx_set_gemm_cta_group(2)
    try:
        test_matmul_forward(oracle, cuda, dt)
        test_matmul_backward(oracle, cuda, dt)
    finally:
        lib.mx_set_gemm_cta_group(1)


SHORT_K = [
    ("keepb-nt", 25640, 600, 256, "k", "k"),      # 201 row tiles (40-row edge), 3 column tiles (88-column edge): 49 CTAs per column tile
    ("keepb-nn", 25640, 600, 256, "k", "mn"),
    ("keepb-tn", 25640, 600, 192, "mn", "mn"),    # three k-blocks: the ring is three slots long
    ("keepb-ragged-k", 25640, 520, 136, "k", "k"),
    ("keepb-one-kb", 151 * 128, 2304, 64, "k", "mn"),
]


@pytest.mark.parametrize("dt", [D.BF16, D.F16], ids=lambda d: d.name)
@pytest.mark.parametrize("case", SHORT_K, ids=lambda c: c[0])
def test_short_reductions_with_the_b_panel_resident(oracle, cuda, dt, case):
    """K <= 256 with many row tiles: the CTAs of a column tile load its B panel once and stream only A.  Against the
    oracle on sampled rows, and bit for bit against the general schedule of the same kernel."""
    from maidenx_b200 import _lib
    lib = _lib.load()
    name, m, n, k, amaj, bmaj = case
    assert lib.mx_debug_gemm_keep_b_ctas((m + 127) // 128, (n + 255) // 256, (k + 63) // 64, 1, 148) > 0
    test_matmul_forward_many_tiles(oracle, cuda, dt, case)
    rng = np.random.default_rng(zlib_seed(name))
    a = H.random_store(rng, dt, m * k, dist="normal")
    b = H.random_store(rng, dt, k * n, dist="normal")
    meta = H.matmul_metadata([m, n], [m, k], [k, n], [k, 1] if amaj == "k" else [1, m], [1, k] if bmaj == "k" else [n, 1], 0, 0)
    kept = H.run_matmul(cuda, dt, meta, m * n, a, b)
    lib.mx_debug_set_gemm_keep_b(0)
    try:
        general = H.run_matmul(cuda, dt, meta, m * n, a, b)
    finally:
        lib.mx_debug_set_gemm_keep_b(1)
    assert np.array_equal(kept, general)


@pytest.mark.parametrize("dt", [D.BF16, D.F16], ids=lambda d: d.name)
@pytest.mark.parametrize("case", [
    # batch, M, N, K, majors, whether A is the same for all batches: rows 16, 32 and 64 bytes off a line, on one side and on both, a ragged side that is copied
    # anyway, slices of a long reduction, and what the rule leaves in place
    (1, 2056, 1544, 1000, "kk", False), (1, 1000, 1032, 1032, "mm", False), (1, 1536, 1544, 1543, "km", False), (1, 520, 1008, 992, "kk", False), (1, 136, 264, 16392, "mk", False),
    (5, 520, 776, 328, "km", False), (7, 264, 520, 200, "kk", True)], ids=lambda c: "x".join(map(str, c)))
def test_operands_off_whole_lines(cuda, dt, case):
    """Copies in whole lines, always and by the rule, change nothing in the sums: bit for bit what the operands give in place; the sums themselves next to float64 (one rounding of an
    f32 sum: half a step of the type and the sum's own error)."""
    from maidenx_b200 import _lib
    lib = _lib.load()
    nb, m, n, k, majors, shared = case
    rng = np.random.default_rng(nb + m + n + k)
    na = 1 if shared else nb
    a, b = H.random_store(rng, dt, na * m * k, dist="normal"), H.random_store(rng, dt, nb * k * n, dist="normal")
    lead = [nb] if nb > 1 else []
    sa, sb = ([0 if shared else m * k] if lead else []) + ([k, 1] if majors[0] == "k" else [1, m]), ([k * n] if lead else []) + ([1, k] if majors[1] == "k" else [n, 1])
    meta = H.matmul_metadata(lead + [m, n], lead + [m, k], lead + [k, n], sa, sb, 0, 0)
    got = {}
    for mode in (0, 2, 1):
        lib.mx_debug_set_gemm_realign(mode)
        try:
            got[mode] = H.run_matmul(cuda, dt, meta, nb * m * n, a, b)
        finally:
            lib.mx_debug_set_gemm_realign(1)
    assert np.array_equal(got[0], got[2]) and np.array_equal(got[0], got[1])
    fa, fb = D.decode(a, dt).astype(np.float64), D.decode(b, dt).astype(np.float64)
    for z in {0, nb - 1}:
        za = fa[(0 if shared else z) * m * k:][:m * k]
        x = za.reshape(m, k) if majors[0] == "k" else za.reshape(k, m).T
        zb = fb[z * k * n:][:k * n]
        y = zb.reshape(n, k).T if majors[1] == "k" else zb.reshape(k, n)
        ref = x @ y
        res = D.decode(got[0], dt).reshape(nb, m, n)[z]
        step = 2.0 ** -8 if dt is D.BF16 else 2.0 ** -11
        assert np.all(np.abs(res - ref) <= step * np.abs(ref) + 2e-5 * np.sqrt(k))


@pytest.mark.parametrize("dt", [D.BF16, D.F16], ids=lambda d: d.name)
@pytest.mark.parametrize("case", [
    # batch, M, N, K, majors, whether A is the same for all batches: edges of row and column tiles, a last k-block that is not full, runs of tiles that end inside a
    # panel; and what the rule leaves to the general schedule
    (97, 600, 760, 256, "kk", True), (149, 641, 504, 200, "km", True), (300, 520, 256, 248, "mm", True), (97, 600, 760, 256, "kk", False), (160, 512, 512, 256, "mm", True),
    (149, 641, 504, 136, "km", True)], ids=lambda c: "x".join(map(str, c)))
def test_short_reductions_of_a_batch_with_the_b_panel_resident(cuda, dt, case):
    """Batched products of K <= 256 that share A load a B panel once for all its row tiles: bit for bit the general schedule, and next to float64 in the first, a middle and the
    last batch (one rounding of an f32 sum: half a step of the type and the sum's own error)."""
    from maidenx_b200 import _lib
    lib = _lib.load()
    nb, m, n, k, majors, shared = case
    rng = np.random.default_rng(nb + m + n + k)
    na = 1 if shared else nb
    a, b = H.random_store(rng, dt, na * m * k, dist="normal"), H.random_store(rng, dt, nb * k * n, dist="normal")
    sa, sb = [0 if shared else m * k, *([k, 1] if majors[0] == "k" else [1, m])], [k * n, *([1, k] if majors[1] == "k" else [n, 1])]
    meta = H.matmul_metadata([nb, m, n], [nb, m, k], [nb, k, n], sa, sb, 0, 0)
    kept = H.run_matmul(cuda, dt, meta, nb * m * n, a, b)
    assert lib.mx_debug_gemm_last_schedule() == (2 if shared and k > 192 and m > 512 else 0)
    lib.mx_debug_set_gemm_keep_b(0)
    try:
        general = H.run_matmul(cuda, dt, meta, nb * m * n, a, b)
        assert lib.mx_debug_gemm_last_schedule() == 0
    finally:
        lib.mx_debug_set_gemm_keep_b(1)
    assert np.array_equal(kept, general)
    got = D.decode(kept, dt).reshape(nb, m, n)
    for i in (0, nb // 2, nb - 1):
        x = D.decode(a.reshape(na, m * k)[0 if shared else i], dt).astype(np.float64)
        y = D.decode(b.reshape(nb, k * n)[i], dt).astype(np.float64)
        x, y = x.reshape(m, k) if majors[0] == "k" else x.reshape(k, m).T, y.reshape(n, k).T if majors[1] == "k" else y.reshape(k, n)
        ref, bound = x @ y, np.abs(x) @ np.abs(y)
        assert np.all(np.abs(got[i] - ref) <= (2.0**-8 if dt.name == "bf16" else 2.0**-11) * np.abs(ref) + k * 2.0**-23 * bound + 2.0**-24)


# ---------------------------------------------------------------------------------------
# Products whose matrices are not 16-byte multiples: operands copied to padded rows, output rows
# written without tensor stores; and the plain tensor-core products that have more than one batch
# dim or are a batched backward.  Bounds: 16-bit results carry one rounding (2^-9 bf16, 2^-11 f16) of an f32 sum;
# f32 the split-tf32 bound of the aligned cases above.
# ---------------------------------------------------------------------------------------
RAGGED = [
    # name, batch dims, M, N, K, a_major, b_major, a_off, b_off
    ("nt-odd", [], 257, 515, 129, "k", "k", 0, 0),
    ("nn-odd", [], 259, 517, 131, "k", "mn", 0, 0),
    ("tn-odd", [], 261, 519, 127, "mn", "mn", 0, 0),
    ("tt-odd", [], 263, 521, 133, "mn", "k", 0, 0),
    ("n-odd", [], 200, 301, 392, "k", "k", 0, 0),             # aligned operands, only the output's rows are ragged
    ("n-even", [], 136, 518, 320, "k", "mn", 0, 0),           # 16-bit rows start on 4 bytes: stores in pairs
    ("k-odd", [], 264, 256, 393, "k", "mn", 0, 0),            # only one operand is copied
    ("offsets", [], 264, 256, 384, "k", "mn", 1, 3),          # regular sizes behind unaligned bases
    ("one-row", [], 1, 4099, 4099, "k", "mn", 0, 0),
    ("narrow", [], 4099, 5, 1001, "k", "k", 0, 0),            # N below one 64-column tile
    ("long-k", [], 33, 65, 9001, "mn", "mn", 0, 0),           # split along K into runs of k-blocks, the last one short
    ("short-split", [], 130, 264, 1032, "k", "k", 0, 0),      # the same on aligned operands, K below the long-reduction plan
    ("batched-odd", [5], 150, 197, 121, "k", "mn", 0, 0),
    ("rank-4", [2, 3], 200, 264, 72, "k", "mn", 0, 0),        # every leading dim is a batch
    ("rank-4-odd", [2, 3], 200, 197, 75, "k", "mn", 0, 0),
    ("wide-batch", [3], 128, 192, 256, "k", "mn", 0, 0),      # 192-column tiles
]


@pytest.mark.parametrize("dt", [D.BF16, D.F16, D.F32], ids=lambda d: d.name)
@pytest.mark.parametrize("case", RAGGED, ids=lambda c: c[0])
def test_products_with_ragged_rows(oracle, cuda, dt, case):
    from oracle import binding
    name, bd, m, n, k, amaj, bmaj, aoff, boff = case
    rng = np.random.default_rng(zlib_seed(name + dt.name))
    cs = H.contiguous_strides
    nb = H.numel(bd) if bd else 1
    a_sh, b_sh, o = [*bd, m, k], [*bd, k, n], [*bd, m, n]
    ast = cs(a_sh) if amaj == "k" else [1, m]
    bst = cs(b_sh) if bmaj == "mn" else [1, k]
    a = H.random_store(rng, dt, nb * m * k + aoff, dist="normal")
    b = H.random_store(rng, dt, nb * k * n + boff, dist="normal")
    meta = H.matmul_metadata(o, a_sh, b_sh, ast, bst, aoff, boff)
    got = H.run_matmul(cuda, dt, meta, nb * m * n, a, b)
    binding.set_wide(True)
    try:
        ref = H.run_matmul(oracle, dt, meta, nb * m * n, a, b)
    finally:
        binding.set_wide(False)
    H.assert_same("matmul", dt, got, ref, float_rel=1e-5 if dt.name == "f32" else 1e-2, what=name, scale=np.sqrt(k))


def _last_f32_form(lib):
    """Slices, CTAs of a cluster, both parts of B in one instruction, columns of a tile: of the thread's last f32 product on the tensor cores."""
    form = (ctypes.c_int * 4)()
    lib.mx_debug_gemm_f32_last_form(form)
    return tuple(form)


@pytest.mark.parametrize("dt", [D.F32], ids=lambda d: d.name)
@pytest.mark.parametrize("case", [
    # M, N, K, majors: two to eight slices, the last one short; ragged rows and edges of tiles; one row and one column of tiles; reductions that are emptied in runs
    (128, 300, 784, "kk"), (128, 784, 300, "km"), (300, 784, 1024, "mm"), (130, 131, 9001, "kk"), (257, 64, 2049, "mk"), (100, 1000, 4100, "km"), (1, 4099, 4099, "km"),
    (512, 72, 8200, "mm"), (1543, 200, 2000, "mm"), (300, 784, 8192, "kk")], ids=lambda c: "x".join(map(str, c)))
def test_slices_summed_in_a_cluster(cuda, dt, case):
    """A split product whose slices are the CTAs of a cluster, next to float64 and to the form with a second launch (the same bits where both cut alike); an
    infinity reaches its own row and nothing else, and nothing is written around the output.  300 x 784 x 8192 takes the form by itself."""
    from maidenx_b200 import _lib, device
    lib = _lib.load()
    m, n, k, majors = case
    rng = np.random.default_rng(m + n + k)
    a, b = (D.encode(rng.standard_normal(x).astype(np.float32).reshape(-1), dt).reshape(x) for x in ((m, k), (k, n)))
    inf = m > 64
    if inf:
        a[m - 1, k // 2] = D.encode(np.array([np.inf], np.float32), dt)[0]
    am, bm = a if majors[0] == "k" else a.T, b.T if majors[1] == "k" else b
    meta = [2, 2, 2, m, n, m, k, k, n, *([k, 1] if majors[0] == "k" else [1, m]), *([1, k] if majors[1] == "k" else [n, 1]), 0, 0]
    guard = 16
    fill = np.full(m * n + 2 * guard, 3, dtype=dt.np_storage)
    got, form = {}, {}
    try:
        for on in (0, 1, 2):
            lib.mx_debug_set_gemm_f32_cluster(on)
            bufs = [device.CudaBuffer.from_host(np.ascontiguousarray(x).reshape(-1)) for x in (am, bm, fill)]
            device.dispatch("matmul", dt.name, meta, m * n, "META", bufs[0].ptr, bufs[1].ptr, bufs[2].ptr + guard * dt.size)
            form[on] = _last_f32_form(lib)
            raw = bufs[2].to_host(dt.np_storage, fill.size)
            assert (raw[:guard] == 3).all() and (raw[-guard:] == 3).all()
            got[on] = D.decode(raw[guard:-guard], dt).astype(np.float64).reshape(m, n)
            for x in bufs:
                x.free()
    finally:
        lib.mx_debug_set_gemm_f32_cluster(1)
    assert form[0][1] == 0 and 2 <= form[2][1] <= 8 and form[2][0] == form[2][1], form
    assert case[:3] != (300, 784, 8192) or form[1][1] > 0, form
    ref = np.matmul(D.decode(a.reshape(-1), dt).astype(np.float64).reshape(m, k)[:m - inf], D.decode(b.reshape(-1), dt).astype(np.float64).reshape(k, n))
    for out in got.values():
        if inf:
            assert np.isinf(out[m - 1]).all()
        err = np.linalg.norm(out[:m - inf] - ref) / np.linalg.norm(ref)
        assert err <= 2e-6, err  # the split product's
    for on in (1, 2):
        if form[on][0] == form[0][0] and form[on][3] == form[0][3]:
            assert np.array_equal(got[on], got[0])


@pytest.mark.parametrize("case", [
    # M, N, K, majors: the shortest reduction of the form, one chunk more and less than whole, a last k-block that is not full; tiles of 64 and 128 columns with edges; no split
    (2048, 1600, 256, "kk"), (1800, 1540, 260, "km"), (2048, 1600, 392, "mm"), (12000, 64, 512, "mk"), (9700, 52, 392, "km"), (2432, 1664, 1000, "km"), (130, 19000, 288, "kk")],
    ids=lambda c: "x".join(map(str, c)))
def test_f32_products_with_both_parts_of_b_in_one_instruction(cuda, case):
    """Next to float64: within the split product's bound, and no further off than the form of three instructions by more than rounding."""
    from maidenx_b200 import _lib, device
    lib = _lib.load()
    m, n, k, majors = case
    rng = np.random.default_rng(m + n + k)
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32)
    am, bm = a if majors[0] == "k" else a.T, b.T if majors[1] == "k" else b
    meta = [2, 2, 2, m, n, m, k, k, n, *([k, 1] if majors[0] == "k" else [1, m]), *([1, k] if majors[1] == "k" else [n, 1]), 0, 0]
    ref = a.astype(np.float64) @ b.astype(np.float64)
    err = []
    try:
        for on in (0, 1):
            lib.mx_debug_set_gemm_f32_wide(on)
            bufs = [device.CudaBuffer.from_host(np.ascontiguousarray(x).reshape(-1)) for x in (am, bm, np.zeros(m * n, np.float32))]
            device.dispatch("matmul", "f32", meta, m * n, "META", bufs[0].ptr, bufs[1].ptr, bufs[2].ptr)
            assert _last_f32_form(lib)[:3] == (1, 0, on) and (n > 64 or _last_f32_form(lib)[3] == 64)
            out = bufs[2].to_host(np.float32, m * n).reshape(m, n)
            err.append(np.linalg.norm(out - ref) / np.linalg.norm(ref))
            for x in bufs:
                x.free()
    finally:
        lib.mx_debug_set_gemm_f32_wide(1)
    assert max(err) <= 2e-6 and err[1] <= 1.02 * err[0], err


@pytest.mark.parametrize("off", [0, 1, 3, 4, 6, 7])
@pytest.mark.parametrize("n", [1, 7, 9, 63, 65, 71, 127, 130, 191, 194, 257, 260, 391])
def test_ragged_output_rows_are_written_whole_and_alone(cuda, n, off):
    """16-bit output rows that start anywhere: cut at the 16-byte boundaries, across the 64-column chunks and the tiles' edges.  Whole
    numbers, so that the result is exact; what lies before and behind the output stays as it was."""
    from maidenx_b200 import device
    m, k = 1100, 256
    rng = np.random.default_rng(n * 8 + off)
    a, b = rng.integers(-2, 3, (m, k)).astype(np.float32), rng.integers(-2, 3, (n, k)).astype(np.float32)
    for dt in (D.BF16, D.F16):
        fill = np.full(m * n + 16, 0x1234, dtype=np.uint16)
        bufs = [device.CudaBuffer.from_host(x) for x in (D.encode(a.reshape(-1), dt), D.encode(b.reshape(-1), dt), fill)]
        device.dispatch("matmul", dt.name, [2, 2, 2, m, n, m, k, k, n, k, 1, 1, k, 0, 0], m * n, "META", bufs[0].ptr, bufs[1].ptr, bufs[2].ptr + 2 * off)
        got = bufs[2].to_host(np.uint16, m * n + 16)
        want = fill.copy()
        want[off:off + m * n] = D.encode((a @ b.T).reshape(-1), dt).view(np.uint16)
        assert np.array_equal(got, want)


@pytest.mark.parametrize("dt", [D.BF16, D.F16, D.F32], ids=lambda d: d.name)
@pytest.mark.parametrize("case", [("batched", [4], 152, 136, 216), ("batched-odd", [4], 151, 133, 219), ("rank-4", [2, 2], 152, 136, 216), ("odd", [], 301, 259, 227),
                                  ("broadcast-b", None, 150, 136, 216)], ids=lambda c: c[0])
def test_batched_and_ragged_backward(oracle, cuda, dt, case):
    from oracle import binding
    name, bd, m, n, k = case
    rng = np.random.default_rng(zlib_seed("bwd" + name + dt.name))
    cs = H.contiguous_strides
    shared = bd is None     # B is one matrix for a batch of four: not a batched product, the reference's index rules apply
    bd = [4] if shared else bd
    nb = H.numel(bd) if bd else 1
    a_sh, b_sh, o = [*bd, m, k], [k, n] if shared else [*bd, k, n], [*bd, m, n]
    nea, neb = H.numel(a_sh), H.numel(b_sh)
    a, b, g = (H.random_store(rng, dt, x, dist="normal") for x in (nea, neb, nb * m * n))
    meta = H.matmul_metadata(o, a_sh, b_sh, cs(a_sh), cs(b_sh), 0, 0)
    got = H.run_matmul_backward(cuda, dt, meta, nea, neb, g, a, b)
    binding.set_wide(True)
    try:
        ref = H.run_matmul_backward(oracle, dt, meta, nea, neb, g, a, b)
    finally:
        binding.set_wide(False)
    for key in ref:
        H.assert_same("matmul_backward", dt, got[key], ref[key], float_rel=1e-5 if dt.name == "f32" else 1e-2, what=f"{name}/{key}", scale=np.sqrt(n if key == "ga" else m))


# ---------------------------------------------------------------------------------------
# Infinities and NaNs in f32 products.  The split into two tf32 parts has no form for them (inf times the zero second part of
# 1.0 would be NaN); the product must give what f32 arithmetic gives.  Every form of the split kernel: aligned, copied and plain-store
# operands, batches, runs along K, 64- and 128-column tiles.
# ---------------------------------------------------------------------------------------
NONFINITE = [
    # name, batch dims, M, N, K, a_major, b_major
    ("aligned", [], 264, 256, 384, "k", "mn"),
    ("aligned-nt", [], 520, 516, 1024, "k", "k"),
    ("aligned-tn", [], 384, 512, 512, "mn", "mn"),
    ("ragged", [], 257, 515, 1031, "k", "k"),
    ("ragged-tt", [], 263, 521, 1033, "mn", "k"),
    ("n-even", [], 200, 514, 1000, "k", "mn"),
    ("narrow", [], 4099, 12, 1001, "k", "k"),
    ("split", [], 130, 264, 4000, "k", "k"),
    ("long-split", [], 132, 264, 8192, "mn", "mn"),
    ("batched", [3], 136, 264, 520, "k", "mn"),
    ("rank-4", [2, 3], 200, 264, 516, "k", "mn"),
]


def special_operands(rng, m, n, k, nb):
    """Mostly values that tf32 holds exactly (small integers, zeros among them), with rows of A and columns of B that hold
    infinities, NaNs of several payloads and both, and one large finite value whose products stay exact."""
    a = rng.integers(-3, 4, (nb, m, k)).astype(np.float32)
    b = rng.integers(-3, 4, (nb, k, n)).astype(np.float32)
    bits = lambda u: np.uint32(u).view(np.float32)  # noqa: E731
    rows, cols = np.arange(0, m, 7), np.arange(3, n, 11)
    for i, v in enumerate((np.inf, -np.inf, bits(0x7F800001), bits(0x7FC00000), bits(0xFF800400), 2.0 ** 20)):
        for z in range(nb):
            if i < len(rows):
                a[z, rows[i], (5 * i + 31 * z) % k] = v
            if i < len(cols):
                b[z, (17 * i + z + k // 2) % k, cols[i]] = v
    a[:, -1, k - 1] = np.inf      # the last row, the last value of K
    b[:, k - 1, -1] = 0.5         # times an exact value
    if m > 20:
        a[:, 20, 0], a[:, 20, k // 2] = np.inf, -np.inf   # inf - inf
        b[:, 0, :] = np.abs(b[:, 0, :]) + 1
    return a, b


@pytest.mark.parametrize("case", NONFINITE, ids=lambda c: c[0])
def test_f32_products_of_infinities_and_nans(oracle, cuda, case):
    """NaN and infinity patterns are those of the f64 product; the finite sums are of integers that f32 holds
    (the bound leaves room for the one product of 2^40 that takes small terms with it)."""
    name, bd, m, n, k, amaj, bmaj = case
    rng = np.random.default_rng(zlib_seed("nonfinite" + name))
    cs = H.contiguous_strides
    nb = H.numel(bd) if bd else 1
    a, b = special_operands(rng, m, n, k, nb)
    with np.errstate(all="ignore"):
        ref = np.matmul(a.astype(np.float64), b.astype(np.float64)).astype(np.float32).reshape(-1)
    a_sh, b_sh, o = [*bd, m, k], [*bd, k, n], [*bd, m, n]
    ast = cs(a_sh) if amaj == "k" else [1, m]
    bst = cs(b_sh) if bmaj == "mn" else [1, k]
    astore = a.reshape(-1) if amaj == "k" else np.ascontiguousarray(a[0].T).reshape(-1)
    bstore = b.reshape(-1) if bmaj == "mn" else np.ascontiguousarray(b[0].T).reshape(-1)
    meta = H.matmul_metadata(o, a_sh, b_sh, ast, bst, 0, 0)
    got = H.run_matmul(cuda, D.F32, meta, nb * m * n, astore, bstore)
    H.assert_same("matmul", D.F32, got, ref, float_rel=1e-5, what=name, scale=np.sqrt(k))


def test_f32_backward_products_of_infinities_and_nans(oracle, cuda):
    for bd, m, n, k in (([4], 264, 272, 280), ([], 301, 519, 227), ([], 264, 512, 256)):
        rng = np.random.default_rng(m)
        cs = H.contiguous_strides
        nb = H.numel(bd) if bd else 1
        g, bt = special_operands(rng, m, k, n, nb)        # grad_a = g . B^T
        bw = np.ascontiguousarray(bt.transpose(0, 2, 1))  # B [k, n]
        a = rng.integers(-2, 3, (nb, m, k)).astype(np.float32)
        a[:, 5, 3] = np.inf
        meta = H.matmul_metadata([*bd, m, n], [*bd, m, k], [*bd, k, n], cs([*bd, m, k]), cs([*bd, k, n]), 0, 0)
        got = H.run_matmul_backward(cuda, D.F32, meta, nb * m * k, nb * k * n, g.reshape(-1), a.reshape(-1), bw.reshape(-1))
        with np.errstate(all="ignore"):
            ra = np.matmul(g.astype(np.float64), bt.astype(np.float64)).astype(np.float32).reshape(-1)
            rb = np.matmul(a.astype(np.float64).transpose(0, 2, 1), g.astype(np.float64)).astype(np.float32).reshape(-1)
        H.assert_same("matmul_backward", D.F32, got["ga"], ra, float_rel=1e-5, what="ga", scale=np.sqrt(n))
        H.assert_same("matmul_backward", D.F32, got["gb"], rb, float_rel=1e-5, what="gb", scale=np.sqrt(m))


@pytest.mark.parametrize("k", [16, 63, 191, 192, 600])
def test_ragged_f32_products_are_no_less_exact_than_f32_sums(cuda, k):
    """Against 64 bits, next to a serial f32 sum with separate multiplies and adds (what the CUDA cores compute).  Below K = 192 the
    two are the same bits; above it the split kernel's error is the smaller one (its parts lose 2^-22 a product, the serial sum half an ulp
    of a growing total a term), 10 % are left for the sample."""
    m, n = 1031, 1031
    for positive in (False, True):
        rng = np.random.default_rng(k)
        a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32)
        if positive:
            a, b = np.abs(a), np.abs(b)
        meta = H.matmul_metadata([m, n], [m, k], [k, n], [k, 1], [n, 1], 0, 0)
        got = H.run_matmul(cuda, D.F32, meta, m * n, a.reshape(-1), b.reshape(-1)).reshape(m, n)
        serial = np.zeros((m, n), np.float32)
        for i in range(k):
            serial += a[:, i:i + 1] * b[i]
        ref = a.astype(np.float64) @ b.astype(np.float64)
        err = lambda x: np.linalg.norm(x - ref) / np.linalg.norm(ref)  # noqa: E731
        assert err(got) <= 1.1 * err(serial), (k, positive, err(got), err(serial))


@pytest.mark.parametrize("dt", [D.BF16, D.F16, D.F32], ids=lambda d: d.name)
@pytest.mark.parametrize("case", [(1, 1, 1 << 20), (1, 1, 65537), (1, 1003, 8200), (1003, 1, 40001), (700, 1, 33000), (3, 5, 40000), (32, 32, 8191), (30, 30, 9001), (4099, 3, 300), (2, 9001, 1003)],
                         ids=lambda c: "x".join(map(str, c)))
def test_vectors_narrow_matrices_and_few_outputs(oracle, cuda, dt, case):
    """One row or column (K-major whatever its strides say), rows of a few elements (copied to 16-byte rows) and few outputs with long
    reductions, on both sides of the line to the block-per-output kernel.  Bounds as above."""
    from oracle import binding
    m, n, k = case
    rng = np.random.default_rng(m + n + k)
    for amaj, bmaj in (("k", "mn"), ("mn", "mn"), ("k", "k")):
        a, b = H.random_store(rng, dt, m * k, dist="normal"), H.random_store(rng, dt, k * n, dist="normal")
        meta = H.matmul_metadata([m, n], [m, k], [k, n], [k, 1] if amaj == "k" else [1, m], [n, 1] if bmaj == "mn" else [1, k], 0, 0)
        got = H.run_matmul(cuda, dt, meta, m * n, a, b)
        binding.set_wide(True)
        try:
            ref = H.run_matmul(oracle, dt, meta, m * n, a, b)
        finally:
            binding.set_wide(False)
        H.assert_same("matmul", dt, got, ref, float_rel=1e-5 if dt.name == "f32" else 1e-2, what=f"{case} {amaj}{bmaj}", scale=np.sqrt(k))


@pytest.mark.parametrize("dt", [D.BF16, D.F16], ids=lambda d: d.name)
@pytest.mark.parametrize("case", [("plain-stores", [], 1290, 1801, 2100, "k", "k"), ("copies", [], 1289, 1800, 3001, "mn", "mn"), ("one-run", [], 1290, 1801, 1024, "k", "k"),
                                  ("one-more", [], 1290, 1801, 1025, "k", "k"), ("batched", [3], 264, 517, 8500, "k", "mn"), ("narrow", [2, 2], 515, 40, 3300, "k", "mn"),
                                  ("split", [], 130, 131, 9001, "k", "k")], ids=lambda c: c[0])
def test_long_sums_of_one_sign_in_16_bit_products(cuda, dt, case):
    """The tensor core's additions truncate; after runs of 1024 (f16) or 4096 (bf16) terms the accumulator is emptied into totals rounded to
    nearest.  Error against 64 bits after the rounding to the type, next to rounding the exact result once.  An instruction adds 16 terms
    and loses at most an ulp, 2^-23, of the accumulator: 64 of them pull by 7.7e-6 of the result, 256 by 3.1e-5.  Next to 2.2e-4 (f16) and 1.8e-3
    (bf16) of the rounding that adds 0.06 and 0.02 % to the error's norm."""
    name, bd, m, n, k, amaj, bmaj = case
    rng = np.random.default_rng(zlib_seed(name))
    cs = H.contiguous_strides
    nb = H.numel(bd) if bd else 1
    a = D.encode((np.abs(rng.standard_normal((nb, m, k))) / np.sqrt(k)).astype(np.float32).reshape(-1), dt)
    b = D.encode((np.abs(rng.standard_normal((nb, k, n))) / np.sqrt(k)).astype(np.float32).reshape(-1), dt)
    av = D.decode(a, dt).astype(np.float64).reshape(nb, m, k)
    bv = D.decode(b, dt).astype(np.float64).reshape(nb, k, n)
    ast, bst = cs([*bd, m, k]), cs([*bd, k, n])
    if amaj == "mn":
        a, ast = np.ascontiguousarray(a.reshape(m, k).T).reshape(-1), [1, m]
    if bmaj == "k" and not bd:
        b, bst = np.ascontiguousarray(b.reshape(k, n).T).reshape(-1), [1, k]
    meta = H.matmul_metadata([*bd, m, n], [*bd, m, k], [*bd, k, n], ast, bst, 0, 0)
    got = D.decode(H.run_matmul(cuda, dt, meta, nb * m * n, a, b), dt).astype(np.float64)
    ref = np.matmul(av, bv).reshape(-1)
    once = D.decode(D.encode(ref.astype(np.float32), dt), dt).astype(np.float64)
    err = lambda x: np.linalg.norm(x - ref) / np.linalg.norm(ref)  # noqa: E731
    assert err(got) <= 1.001 * err(once), (err(got), err(once))
    assert abs(((got - once) / ref).mean()) < (64 if dt.name == "f16" else 256) * 2.0 ** -23 + 4 * err(once) / np.sqrt(ref.size)


@pytest.mark.parametrize("dt", [D.F32, D.F64, D.BF16, D.I32, D.U8], ids=lambda d: d.name)
@pytest.mark.parametrize("case", [(4001, 1, 1, 16), (4001, 1, 17, 5), (9000, 3, 2, 7), (5000, 5, 3, 33), (3000, 2, 65, 4), (2500, 7, 9, 1), (700, 1, 1, 3), (64, 63, 3, 1)], ids=lambda c: "x".join(map(str, c)))
def test_many_small_batches(oracle, cuda, dt, case):
    """Tiles of 64 rows that span batches (few rows a batch, short reductions) and blocks of one batch each: both add in the
    element-type loop's order, so f32, f64 and integers are bit-exact, and 16-bit types round one f32 sum."""
    from oracle import binding
    nb, m, n, k = case
    rng = np.random.default_rng(nb + k)
    cs = H.contiguous_strides
    shapes = [nb, m, k], [nb, k, n], [nb, m, n]
    a, b, g = (_inputs(rng, dt, H.numel(x)) for x in shapes)
    binding.set_wide(dt.name == "bf16")
    try:
        for bst in (cs(shapes[1]), [0, n, 1]):        # every batch its own B, and one for all
            meta = H.matmul_metadata(shapes[2], shapes[0], shapes[1], cs(shapes[0]), bst, 0, 0)
            ref = H.run_matmul(oracle, dt, meta, nb * m * n, a, b)
            H.assert_same("matmul", dt, H.run_matmul(cuda, dt, meta, nb * m * n, a, b), ref, what=str(bst))
        meta = H.matmul_metadata(shapes[2], shapes[0], shapes[1], cs(shapes[0]), cs(shapes[1]), 0, 0)
        ref = H.run_matmul_backward(oracle, dt, meta, nb * m * k, nb * k * n, g, a, b)
        got = H.run_matmul_backward(cuda, dt, meta, nb * m * k, nb * k * n, g, a, b)
    finally:
        binding.set_wide(False)
    for key in ref:
        H.assert_same("matmul_backward", dt, got[key], ref[key], what=key)


@pytest.mark.parametrize("dt", [D.BF16, D.F32], ids=lambda d: d.name)
@pytest.mark.parametrize("case", [(256, 256, 8192), (128, 264, 1536)], ids=lambda c: "x".join(map(str, c)))
def test_split_products_under_capture(cuda, dt, case):
    """A product with few tiles is cut along K in a graph as it is in a direct call: the same bits, also after the thread's scratch block
    has been replaced by a larger one."""
    import ctypes

    import torch

    from maidenx_b200 import _lib

    lib, m, n, k = _lib.load(), *case
    tdt = {"bf16": torch.bfloat16, "f32": torch.float32}[dt.name]
    g = torch.Generator(device="cuda").manual_seed(5)
    a, b = torch.randn(m, k, device="cuda", generator=g).to(tdt), torch.randn(k, n, device="cuda", generator=g).to(tdt)
    meta = np.asarray(H.matmul_metadata([m, n], [m, k], [k, n], [k, 1], [n, 1], 0, 0), dtype=np.uint64)
    direct, replayed = torch.zeros(m, n, device="cuda", dtype=tdt), torch.zeros(m, n, device="cuda", dtype=tdt)
    op = _lib.op("matmul", dt.name)
    call = lambda out: op(ctypes.c_size_t(m * n), meta.ctypes.data, a.data_ptr(), b.data_ptr(), out.data_ptr())  # noqa: E731
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    lib.mx_set_stream(s.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    try:
        call(direct)
        s.synchronize()
        with torch.cuda.graph(graph, stream=s):
            call(replayed)
        for round_ in range(2):
            replayed.zero_()
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            assert lib.mx_last_error() == 0
            assert torch.equal(direct.view(torch.uint8), replayed.view(torch.uint8)), round_
            # a fold with wide partial results of its own: the block grows
            x = torch.ones(2, 9, 3000, 4, 700, device="cuda")
            out = torch.zeros(9, 700, device="cuda")
            fold = np.asarray([2, 9, 3000, 4, 700, 9 * 3000 * 4 * 700, 3000 * 4 * 700, 4 * 700, 700, 1, 1, 9, 1, 1, 700, 0], dtype=np.uint64)
            _lib.op("sum_to_shape", "f32")(ctypes.c_size_t(x.numel()), ctypes.c_size_t(5), fold.ctypes.data, x.data_ptr(), out.data_ptr())
            big = torch.ones(8, 400000, 16, device="cuda")
            kept = torch.zeros(400000, device="cuda")
            fold2 = np.asarray([8, 400000, 16, 6400000, 16, 1, 1, 400000, 1, 0], dtype=np.uint64)
            _lib.op("sum_to_shape", "f32")(ctypes.c_size_t(big.numel()), ctypes.c_size_t(3), fold2.ctypes.data, big.data_ptr(), kept.data_ptr())
            s.synchronize()
            assert float(out[0, 0]) == 2 * 3000 * 4 and float(kept[7]) == 128.0
    finally:
        lib.mx_set_stream(None)
        del graph


# batch, M, N, K, majors, operand shared by the batch, base offset in elements: edges of tiles and of scales' blocks (128 values of K, 64 of a k-block), a lone k-block,
# slices of a long reduction, batches, ragged rows and bases
PAIRS = [(1, 384, 384, 128, "kk", "", 0), (1, 385, 260, 196, "km", "", 0), (1, 516, 532, 64, "mm", "", 0), (1, 132, 136, 4100, "mk", "", 0), (5, 256, 200, 320, "km", "a", 0),
         (6, 160, 256, 448, "kk", "b", 0), (9, 130, 132, 200, "mm", "", 0), (1, 257, 331, 333, "kk", "", 0), (1, 131, 257, 1001, "mm", "", 1), (3, 129, 233, 205, "km", "a", 0)]


def _pairs_product(cuda, lib, case, a, b, mode):
    nb, m, n, k, majors, shared, off = case
    lead = [nb] if nb > 1 else []
    sa = ([0 if "a" in shared else m * k] if lead else []) + ([k, 1] if majors[0] == "k" else [1, m])
    sb = ([0 if "b" in shared else k * n] if lead else []) + ([1, k] if majors[1] == "k" else [n, 1])
    lib.mx_debug_set_gemm_f32_pairs(mode)
    try:
        got = H.run_matmul(cuda, D.F32, H.matmul_metadata(lead + [m, n], lead + [m, k], lead + [k, n], sa, sb, off, off), nb * m * n, a, b)
        return got.reshape(nb, m, n), lib.mx_debug_gemm_f32_last_pairs()
    finally:
        lib.mx_debug_set_gemm_f32_pairs(1)


def _pairs_operands(case, rng, dist):
    nb, m, n, k, majors, shared, off = case
    draw = (lambda s: rng.standard_normal(s)) if dist == "normal" else (lambda s: rng.random(s))
    a, b = (draw(off + (1 if s in shared else nb) * r * k).astype(np.float32) for s, r in (("a", m), ("b", n)))
    x = a[off:].reshape(-1, m, k) if majors[0] == "k" else a[off:].reshape(-1, k, m).transpose(0, 2, 1)
    y = b[off:].reshape(-1, n, k).transpose(0, 2, 1) if majors[1] == "k" else b[off:].reshape(-1, k, n)
    return a, b, x, y


@pytest.mark.parametrize("dist", ["normal", "positive"])
@pytest.mark.parametrize("case", PAIRS, ids=lambda c: "x".join(map(str, c)))
def test_f32_products_as_pairs_of_f16(cuda, case, dist):
    """Next to float64, relative to the sums' size: 2^-23 of each factor, a truncation of at most 2^-24 of the running sum for each of a chunk's eight instructions, the totals' own
    rounding - and no further from float64 than the tf32 kernel (a tenth for chance)."""
    from maidenx_b200 import _lib
    lib = _lib.load()
    a, b, x, y = _pairs_operands(case, np.random.default_rng(sum(case[:4])), dist)
    ref = x.astype(np.float64) @ y.astype(np.float64)
    err = {}
    ragged = any(v % 4 for v in ((case[3] if case[4][0] == "k" else case[1]), case[2], case[6])) or (case[4][1] == "k" and case[3] % 4)
    for mode in (0, 2, 3):
        got, pairs = _pairs_product(cuda, lib, case, a, b, mode)
        assert (pairs > 0) == (mode > 0)
        err[mode] = np.linalg.norm(got - ref) / np.linalg.norm(ref)
    assert err[2] < 6e-7 and err[3] < 3e-7
    assert err[3 if ragged else 2] <= 1.1 * err[0]


@pytest.mark.parametrize("case", [(2048, 1600, 256, "kk"), (1800, 1540, 260, "km"), (2048, 1600, 392, "mm"), (2432, 1664, 1000, "km")], ids=lambda c: "x".join(map(str, c)))
def test_the_tf32_kernel_s_forms_where_pairs_are_faster(cuda, case):
    from maidenx_b200 import _lib
    lib = _lib.load()
    lib.mx_debug_set_gemm_f32_pairs(0)
    try:
        test_f32_products_with_both_parts_of_b_in_one_instruction(cuda, case)
    finally:
        lib.mx_debug_set_gemm_f32_pairs(1)


@pytest.mark.parametrize("what", ["tiny", "tiny_k", "huge", "small_all", "denormal", "inf", "nan", "zeros"])
@pytest.mark.parametrize("case", [(1, 300, 260, 400, "km", "", 0), (4, 132, 136, 260, "kk", "a", 0), (1, 257, 231, 333, "kk", "", 0)], ids=lambda c: "x".join(map(str, c)))
def test_operands_that_are_not_fit_for_pairs(cuda, case, what):
    """Elements far below their block's largest, blocks out of range, infinities and NaNs: the result is the tf32 kernel's, launched behind the pairs, bit for bit.  Zeros are fit."""
    from maidenx_b200 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(7)
    a, b, x, y = _pairs_operands(case, rng, "normal")
    k, off = case[3], case[6]
    if what == "tiny":  # all of one row of A, which only a block's common scale would lose
        a[off:off + k] *= np.float32(1e-13)
    elif what == "tiny_k":  # every third value of K, made up for in B
        x[:, :, ::3] *= np.float32(1e12)
        y[:, ::3] *= np.float32(1e-12)
    elif what == "huge":
        a[off + 5], b[off + 7] = 3e38, 1e-37
    elif what == "small_all":
        a *= np.float32(1e-20)
    elif what == "denormal":
        a[off + 3] = 1e-42
    elif what == "inf":
        a[off + 1], b[off + 2 * k + 1] = np.inf, -np.inf
    elif what == "nan":
        b[off + 11] = np.nan
    else:
        a[off:off + 200 * 64] = 0.0
    got, pairs = _pairs_product(cuda, lib, case, a, b, 2)
    want, _ = _pairs_product(cuda, lib, case, a, b, 0)
    assert pairs > 0 and np.array_equal(got, want, equal_nan=True) == (what != "zeros")
    with np.errstate(all="ignore"):
        ref = x.astype(np.float64) @ y.astype(np.float64)
        size = np.abs(x).astype(np.float64) @ np.abs(y).astype(np.float64)
    fine = np.isfinite(want) & np.isfinite(ref)
    assert np.all(np.abs(got[fine] - ref[fine]) <= 4e-6 * size[fine] + 1e-42)


@pytest.mark.parametrize("where", ["rows", "k"])
@pytest.mark.parametrize("depth", [20, 27, 28, 29, 30, 32])
@pytest.mark.parametrize("majors", ["kk", "mm"])
def test_elements_far_below_their_block_s_largest(cuda, majors, depth, where):
    """A product that selects elements gives each of them to 2^-22, as the tf32 kernel does, however small it is next to its neighbours: 2^-23 as pairs (h1 normal), or left to that kernel."""
    from maidenx_b200 import _lib
    m, k, n = 320, 256, 256
    rng = np.random.default_rng(depth)
    x = ((rng.random((m, k)) + 1) * rng.choice([-1, 1], (m, k))).astype(np.float32)
    x[(slice(1, None, 3),) if where == "rows" else (slice(None), slice(1, None, 3))] *= np.float32(2.0 ** -depth)
    y = np.eye(k, n, dtype=np.float32)
    a, b = (x if majors[0] == "k" else x.T.copy()).ravel(), y.ravel()
    got, pairs = _pairs_product(cuda, _lib.load(), (1, m, n, k, majors, "", 0), a, b, 2)
    assert pairs > 0 and np.all(np.abs(got[0] - x) <= 2.0 ** -22 * np.abs(x))


@pytest.mark.parametrize("batch,fan_in,fan_out", [(550, 192, 630), (596, 53, 3816), (880, 43, 792), (504, 24, 3087), (91, 4000, 200)], ids=str)
def test_short_f32_products_run_without_the_launches_of_pairs(cuda, batch, fan_in, fan_out):
    """Layers whose products take less than the host takes for a split pass, a product in pairs and a kernel behind it stay with one kernel; products of several times that run as pairs."""
    from maidenx_b200 import _lib
    lib = _lib.load()

    def ran_as_pairs(m, n, k, majors):
        _pairs_product(cuda, lib, (1, 256, 256, 512, "kk", "", 0), np.ones(1 << 17, np.float32), np.ones(1 << 17, np.float32), 0)
        return _pairs_product(cuda, lib, (1, m, n, k, majors, "", 0), np.ones(m * k, np.float32), np.ones(n * k, np.float32), 1)[1] > 0

    assert not ran_as_pairs(batch, fan_out, fan_in, "kk") and not ran_as_pairs(batch, fan_in, fan_out, "km") and not ran_as_pairs(fan_out, fan_in, batch, "mm")
    assert ran_as_pairs(2048, 2048, 1024, "kk") and ran_as_pairs(2100, 1500, 1001, "km")


def test_a_large_product_in_pairs_stays_within_the_pool(cuda):
    """Ragged operands of 392 MB: the pairs and the copies of the kernel behind them share their memory, so that the next call finds all of it in the pool and maps none."""
    import torch

    from maidenx_b200 import _lib, device
    lib, (m, n, k) = _lib.load(), (6065, 12, 16147)
    a, b, out = torch.ones(m, k, device="cuda"), torch.ones(n, k, device="cuda"), torch.empty(m, n, device="cuda")
    lib.mx_debug_set_gemm_f32_pairs(2)
    try:
        for _ in range(3):
            torch.cuda.synchronize()
            before = torch.cuda.mem_get_info()[0]
            device.dispatch("matmul", "f32", H.matmul_metadata([m, n], [m, k], [k, n], [k, 1], [1, k], 0, 0), m * n, "META", a.data_ptr(), b.data_ptr(), out.data_ptr())
            mapped = before - torch.cuda.mem_get_info()[0]
        assert lib.mx_debug_gemm_f32_last_pairs() > 0 and mapped < 64 << 20
        assert bool((out == k).all())
    finally:
        lib.mx_debug_set_gemm_f32_pairs(1)


# products that are cut along K as pairs and by the tf32 kernel, by the latter alone, into a cluster; ragged
@pytest.mark.parametrize("case,slices", [((1, 512, 512, 8192, "kk", "", 0), "both"), ((1, 300, 261, 9001, "km", "", 1), "both"), ((1, 400, 400, 256, "kk", "", 0), "tf32"),
                                         ((1, 300, 784, 8192, "kk", "", 0), "cluster")], ids=str)
def test_the_kernel_behind_the_gate_is_cut_along_k(cuda, case, slices):
    """A product that is not fit for pairs runs in the form, and to the bits, that it has without them; the same product with fit operands is the pairs' own sum."""
    import ctypes

    from maidenx_b200 import _lib
    lib, form = _lib.load(), (ctypes.c_int * 4)()
    a, b, x, y = _pairs_operands(case, np.random.default_rng(3), "normal")
    got, pairs = _pairs_product(cuda, lib, case, a, b, 2)
    lib.mx_debug_gemm_f32_last_form(form)
    assert (pairs > 1) == (slices in ("both", "cluster")) and form[0] > 1 and (form[1] > 0) == (slices == "cluster")
    ref = x.astype(np.float64) @ y.astype(np.float64)
    assert np.linalg.norm(got - ref) < 6e-7 * np.linalg.norm(ref)
    a[case[6] + 5] = np.float32(1e-13)  # below 2^-40 of its neighbours
    got, pairs = _pairs_product(cuda, lib, case, a, b, 2)
    want, _ = _pairs_product(cuda, lib, case, a, b, 0)
    assert pairs > 0 and np.array_equal(got, want)


@pytest.mark.parametrize("case", [(512, 512, 8192), (768, 768, 16384), (512, 1024, 4096)], ids=str)
def test_products_in_pairs_are_cut_along_k_under_capture(cuda, case):
    """There is no workspace for pairs in a graph: a product that runs as pairs in a direct call runs there in the tf32 kernel, cut along K and with the bits of a direct call of that kernel,
    although the thread has made no other call that left it a scratch block."""
    import ctypes
    import threading

    import torch

    from maidenx_b200 import _lib
    lib, (m, n, k) = _lib.load(), case
    g = torch.Generator(device="cuda").manual_seed(5)
    a, b = torch.randn(m, k, device="cuda", generator=g), torch.randn(n, k, device="cuda", generator=g)
    meta = np.asarray(H.matmul_metadata([m, n], [m, k], [k, n], [k, 1], [1, k], 0, 0), dtype=np.uint64)
    direct, replayed, tf32 = (torch.zeros(m, n, device="cuda") for _ in range(3))
    call = lambda out: _lib.op("matmul", "f32")(ctypes.c_size_t(m * n), meta.ctypes.data, a.data_ptr(), b.data_ptr(), out.data_ptr())  # noqa: E731
    seen = {}

    def new_thread():
        form, s = (ctypes.c_int * 4)(), torch.cuda.Stream()
        lib.mx_set_stream(s.cuda_stream)
        graph = torch.cuda.CUDAGraph()
        call(direct)
        s.synchronize()
        seen["pairs"] = lib.mx_debug_gemm_f32_last_pairs()
        with torch.cuda.graph(graph, stream=s):
            call(replayed)
        lib.mx_debug_gemm_f32_last_form(form)
        seen["slices"] = form[0]
        graph.replay()
        torch.cuda.synchronize()
        lib.mx_debug_set_gemm_f32_pairs(0)
        call(tf32)
        s.synchronize()
        lib.mx_set_stream(None)

    lib.mx_debug_set_gemm_f32_pairs(2)
    try:
        t = threading.Thread(target=new_thread)
        t.start()
        t.join()
    finally:
        lib.mx_debug_set_gemm_f32_pairs(1)
    assert seen["pairs"] > 0 and seen["slices"] > 1 and torch.equal(replayed, tf32)
    assert float((direct - replayed).norm() / replayed.norm()) < 1e-6


@pytest.mark.parametrize("m,n,k,copies", [(336, 8, 11560, 0), (224, 32, 10248, 0), (24, 24, 10592, 0), (200, 8, 6896, 0), (544, 680, 168, 0), (2504, 2480, 3688, 3)], ids=str)
def test_which_operands_off_whole_lines_are_copied(cuda, m, n, k, copies):
    """Few tiles, whose slices of K run side by side, and short reductions are read in place; many tiles of a long reduction are worth the copies."""
    from maidenx_b200 import _lib
    rng = np.random.default_rng(0)
    a, b = (D.encode(rng.standard_normal(s), D.BF16) for s in (m * k, n * k))
    got = H.run_matmul(cuda, D.BF16, H.matmul_metadata([m, n], [m, k], [k, n], [k, 1], [1, k], 0, 0), m * n, a, b)
    assert _lib.load().mx_debug_gemm_last_copies() == copies
    ref = D.decode(a, D.BF16).reshape(m, k).astype(np.float64) @ D.decode(b, D.BF16).reshape(n, k).T.astype(np.float64)
    assert np.all(np.abs(D.decode(got, D.BF16).reshape(m, n) - ref) <= 2.0 ** -8 * np.abs(ref) + 2.0 ** -22 * k)


@pytest.mark.parametrize("m,n,k,copies", [(8, 3136, 400, 1), (40, 3136, 400, 0), (3136, 40, 320, 2)], ids=str)
def test_which_operands_of_short_mn_major_rows_are_copied(cuda, m, n, k, copies):
    """Rows of K of few elements, read by many tiles of a batch that shares them: what was measured to be the faster way."""
    from maidenx_b200 import _lib
    rng, batch = np.random.default_rng(1), 32
    a_b, b_b = (0, k * n) if m < n else (m * k, 0)
    a, b = (D.encode(rng.standard_normal(s), D.BF16) for s in ((batch if a_b else 1) * m * k, (batch if b_b else 1) * n * k))
    a_st = [1, m] if m < n else [k, 1]
    meta = H.matmul_metadata([batch, m, n], [batch, m, k], [batch, k, n], [a_b, *a_st], [b_b, n, 1], 0, 0)
    got = H.run_matmul(cuda, D.BF16, meta, batch * m * n, a, b)
    assert _lib.load().mx_debug_gemm_last_copies() == copies
    x = np.broadcast_to(D.decode(a, D.BF16).reshape((-1, k, m) if m < n else (-1, m, k)), (batch, k, m) if m < n else (batch, m, k)).astype(np.float32)
    y = np.broadcast_to(D.decode(b, D.BF16).reshape(-1, k, n), (batch, k, n)).astype(np.float32)
    ref = ((x.transpose(0, 2, 1) if m < n else x) @ y).astype(np.float64)
    assert np.all(np.abs(D.decode(got, D.BF16).reshape(batch, m, n) - ref) <= 2.0 ** -8 * np.abs(ref) + 2.0 ** -18 * k)


def test_large_workspaces_of_two_sizes_find_each_other_s_block(cuda):
    """Products whose workspaces are 392 and 401 MB, in turn behind a synchronisation: the larger one's block serves both, and no call maps memory."""
    import torch

    from maidenx_b200 import _lib, device
    lib, n, k = _lib.load(), 12, 16147
    a, b, out = torch.ones(6200, k, device="cuda"), torch.ones(n, k, device="cuda"), torch.empty(6200, n, device="cuda")
    lib.mx_debug_set_gemm_f32_pairs(2)
    try:
        for _ in range(3):
            torch.cuda.synchronize()
            before = torch.cuda.mem_get_info()[0]
            for m in (6065, 6200):
                device.dispatch("matmul", "f32", H.matmul_metadata([m, n], [m, k], [k, n], [k, 1], [1, k], 0, 0), m * n, "META", a.data_ptr(), b.data_ptr(), out.data_ptr())
                assert lib.mx_debug_gemm_f32_last_pairs() > 0
            mapped = before - torch.cuda.mem_get_info()[0]
        assert mapped < 64 << 20 and bool((out == k).all())
    finally:
        lib.mx_debug_set_gemm_f32_pairs(1)
