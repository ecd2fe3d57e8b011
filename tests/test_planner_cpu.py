"""The host-side launch planners, without a GPU: layouts of the benchmark and of the parity tests must be
recognised as the kernel class that was written for them (a silent fall to the generic gather kernel would keep
every parity test green and lose an order of magnitude of bandwidth)."""
import ctypes

import numpy as np

import harness as H
from maidenx_b200 import _lib

FLAT, ROW, TILE, GENERIC, SERIAL, FLAT_SHIFT = 1, 2, 3, 4, 5, 7
ROWS, COLS, SCATTER = 1, 2, 3
BASE = 0x7F0000000000  # a 256-byte aligned pretend device address: the planner only looks at alignment


def ew_plan(meta, nd, n, nin=2, inplace=False, esz=4, osz=4, out=BASE, a=BASE + (1 << 32), b=BASE + (2 << 32)):
    lib = _lib.load()
    m = np.asarray(meta, dtype=np.uint64)
    rank, vec, tmask = ctypes.c_int(), ctypes.c_int(), ctypes.c_int()
    kind = lib.mx_debug_elementwise_plan(n, nd, m.ctypes.data, nin, int(inplace), esz, osz, out, a, b, ctypes.byref(rank), ctypes.byref(vec),
                                         ctypes.byref(tmask))
    return kind, rank.value, vec.value, tmask.value


def test_benchmark_layouts_take_their_kernels():
    R = C = 16384
    n = R * C
    assert ew_plan([R, C, C, 1, C, 1, 0, 0], 2, n)[:3] == (FLAT, 1, 1)                 # contiguous: merged to one dim
    kind, rank, vec, tmask = ew_plan([R, C, 1, R, C, 1, 0, 0], 2, n)                    # transposed lhs
    assert (kind, vec, tmask) == (TILE, 1, 1)
    assert ew_plan([R, C, C, 1, 0, 1, 0, 0], 2, n)[:3] == (ROW, 2, 1)                  # rhs broadcast from [1, C]
    assert ew_plan([R, C, 1, R, 0], 2, n, nin=1)[0] == TILE                            # unary on a transposed view
    assert ew_plan([R, C, 0, 1, 0], 2, n, nin=1)[0] == ROW                             # unary on a broadcast row
    for esz in (2, 4, 8):
        assert ew_plan([R, C, 1, R, C, 1, 0, 0], 2, n, esz=esz, osz=esz)[0] == TILE


def test_odd_layouts_degrade_gracefully():
    # offset 1 (the layout of the reference's test fixtures) breaks 16-byte alignment: the call takes the flat kernel's
    # shifted form (aligned 16-byte loads + funnel shift), not the per-element gather
    assert ew_plan([1000, 1, 1, 1, 1], 1, 1000)[:3] == (FLAT_SHIFT, 1, 1)
    # the same view at an aligned offset is flat again
    assert ew_plan([1000, 1, 1, 4, 8], 1, 1000)[:3] == (FLAT, 1, 1)
    # a permuted 3-d view has no unit-stride pairing the tile kernel handles
    assert ew_plan([5, 6, 7, 1, 35, 5, 42, 7, 1, 0, 0], 3, 210)[0] == GENERIC
    # size-1 dims are dropped before anything else
    assert ew_plan([1, 9, 1, 11, 99, 11, 11, 1, 99, 11, 11, 1, 0, 0], 4, 99)[:2] == (FLAT, 1)
    # both operands transposed the same way: the output is the only direct operand
    kind, _, _, tmask = ew_plan([96, 80, 1, 96, 1, 96, 0, 0], 2, 96 * 80)
    assert (kind, tmask) == (TILE, 3)
    # in-place with an lhs that overlaps itself (stride 0) must run serially
    assert ew_plan([8, 4, 0, 1, 4, 1, 0, 0], 2, 32, inplace=True, out=BASE, a=BASE)[0] == SERIAL
    # scalars
    assert ew_plan([2, 1], 0, 1)[0] in (FLAT, GENERIC)


def red_plan(meta, nd, nr, n, shape=False):
    lib = _lib.load()
    m = np.asarray(meta, dtype=np.uint64)
    o, r, i = ctypes.c_size_t(), ctypes.c_size_t(), ctypes.c_size_t()
    kind = lib.mx_debug_reduce_plan(n, nd, nr, m.ctypes.data, int(shape), ctypes.byref(o), ctypes.byref(r), ctypes.byref(i))
    return kind, o.value, r.value, i.value


def test_reduction_layouts_take_their_kernels():
    R, C = 8192, 16384
    n = R * C
    assert red_plan([R, C, C, 1, R, C, 0], 2, 1, n) == (COLS, 1, R, C)                  # dim 0: fold 8192 rows of 16384 columns
    assert red_plan([R, C, C, 1, C, 1, 0], 2, 1, n)[:3] == (ROWS, R, C)                 # dim 1: 8192 rows of 16384
    # sum_to_shape [64, 512, 4096] -> [1, 1, 4096]: the two leading dims fold into one reduced extent
    assert red_plan([64, 512, 4096, 512 * 4096, 4096, 1, 1, 1, 4096, 0], 3, 0, 64 * 512 * 4096, shape=True) == (COLS, 1, 64 * 512, 4096)
    # the middle dim of a 3-d tensor
    assert red_plan([7, 129, 5, 645, 5, 1, 129, 5, 0], 3, 1, 7 * 129 * 5) == (COLS, 7, 129, 5)
    # a full reduction as the MLP's bias gradient issues it
    assert red_plan([1 << 20, 1, 1 << 20, 1, 0], 1, 1, 1 << 20)[:3] == (ROWS, 1, 1 << 20)
    # two reduced dims at once, or a transposed input, follow the reference's index formulas literally
    assert red_plan([4, 6, 8, 48, 8, 1, 4, 8, 48, 1, 0], 3, 2, 192)[0] == SCATTER
    assert red_plan([64, 32, 1, 64, 64, 1, 0], 2, 1, 2048)[0] == SCATTER


def mm_path(meta, num_els, a=BASE, b=BASE + (1 << 32), out=BASE + (2 << 32), f32=False):
    lib = _lib.load()
    m_ = np.asarray(meta, dtype=np.uint64)
    amn, bmn = ctypes.c_int(-1), ctypes.c_int(-1)
    M, N, K = ctypes.c_size_t(), ctypes.c_size_t(), ctypes.c_size_t()
    fn = lib.mx_debug_matmul_forward_path_f32 if f32 else lib.mx_debug_matmul_forward_path
    tc = fn(num_els, m_.ctypes.data, a, b, out, ctypes.byref(amn), ctypes.byref(bmn), ctypes.byref(M),
                                          ctypes.byref(N), ctypes.byref(K))
    return tc, amn.value, bmn.value, M.value, N.value, K.value


def test_the_three_products_of_a_linear_layer_run_on_the_tensor_core_kernel():
    """Forward x . W^T (B read through a transposed view), dW = du^T . a (A through a transposed view) and
    dX = du . W (both dense), at the benchmark's per-rank shapes for 1 and 8 ranks: none needs a transposed copy."""
    D = 8192
    for B in (16384, 2048):
        assert mm_path([2, 2, 2, B, D, B, D, D, D, D, 1, 1, D, 0, 0], B * D) == (1, 0, 0, B, D, D)       # NT: both K-major
        assert mm_path([2, 2, 2, D, D, D, B, B, D, 1, D, D, 1, 0, 0], D * D) == (1, 1, 1, D, D, B)       # TN: both MN-major
        assert mm_path([2, 2, 2, B, D, B, D, D, D, D, 1, D, 1, 0, 0], B * D) == (1, 0, 1, B, D, D)       # NN


def mm_plan(dt, out_shape, a_shape, b_shape, ast=None, bst=None, aoff=0, boff=0, which=0, out=BASE + (2 << 32)):
    """(batches, operand majors, M, N, K, prepared) of a product; dt "f32" or a 16-bit type.  prepared: 1 / 2 = first / second operand
    copied, 4 / 8 = output without tensor stores, element-wise / in pairs."""
    lib = _lib.load()
    esz = 4 if dt == "f32" else 2
    meta = np.asarray(H.matmul_metadata(out_shape, a_shape, b_shape, ast or H.contiguous_strides(a_shape), bst or H.contiguous_strides(b_shape), aoff, boff),
                      dtype=np.uint64)
    amn, bmn, prep = ctypes.c_int(-1), ctypes.c_int(-1), ctypes.c_int(-1)
    M, N, K = ctypes.c_size_t(), ctypes.c_size_t(), ctypes.c_size_t()
    a, b = BASE, BASE + (1 << 32)
    x, y = {0: (a, b), 1: (a, b + boff * esz), 2: (a, b + aoff * esz)}[which]   # backward calls pass g and the other operand's first element
    tc = lib.mx_debug_matmul_plan(esz, which, H.numel(out_shape), H.numel(a_shape), H.numel(b_shape), meta.ctypes.data, x, y, out, ctypes.byref(amn),
                                  ctypes.byref(bmn), ctypes.byref(M), ctypes.byref(N), ctypes.byref(K), ctypes.byref(prep))
    return (tc, amn.value, bmn.value, M.value, N.value, K.value, prep.value) if tc else 0


def test_products_the_tensor_core_kernel_does_not_take():
    assert mm_path([2, 2, 2, 64, 64, 64, 64, 64, 64, 64, 1, 64, 1, 0, 0], 64 * 64)[0] == 0               # too small for a persistent launch
    assert mm_path([2, 2, 2, 512, 512, 512, 512, 512, 512, 1024, 2, 512, 1, 0, 0], 512 * 512)[0] == 0    # A with a stride of 2 along k
    assert mm_path([3, 3, 3, 4, 512, 512, 4, 512, 512, 4, 512, 512, 262144, 512, 1, 262144, 512, 1, 0, 0], 4 * 512 * 512)[0] == 4  # batched rank-3: one launch, four batches
    # batches of one operand that are not whole matrices apart cannot be copied; in place they only need 16-byte strides
    cs = [512 * 512 + 8, 512, 1]
    assert mm_plan("bf16", [3, 512, 512], [3, 512, 512], [3, 512, 512], ast=cs)[0] == 3
    assert mm_plan("bf16", [3, 512, 511], [3, 512, 512], [3, 512, 511], ast=cs) == 0
    assert mm_plan("bf16", [4, 512, 512], [1, 512, 512], [4, 512, 511 + 1], aoff=1) == 0   # a size-1 batch dim: the copy would read four batches
    assert mm_plan("bf16", [4, 512, 512], [4, 512, 512], [512, 512], which=2) == 0        # b shared by the batch: not a batched product


def test_products_that_are_prepared_for_the_tensor_core_kernel():
    """Operands whose rows or bases are not 16-byte multiples are copied (1, 2), output rows like that written without tensor stores
    (4 element-wise, 8 in pairs); batches of any rank and batched backward products need nothing."""
    assert mm_plan("bf16", [512, 516], [512, 512], [512, 516]) == (1, 0, 1, 512, 516, 512, 2 | 8)
    assert mm_plan("bf16", [512, 515], [512, 512], [512, 515]) == (1, 0, 1, 512, 515, 512, 2 | 4)
    assert mm_plan("bf16", [512, 516], [512, 512], [512, 516], bst=[1, 512]) == (1, 0, 0, 512, 516, 512, 8)
    assert mm_plan("f16", [512, 512], [512, 512], [512, 512], aoff=1) == (1, 0, 1, 512, 512, 512, 1)
    assert mm_plan("f16", [512, 512], [512, 512], [512, 512], out=BASE + 2) == (1, 0, 1, 512, 512, 512, 4)
    assert mm_plan("f32", [512, 514], [512, 512], [512, 514]) == (1, 0, 1, 512, 514, 512, 2 | 8)
    assert mm_plan("f32", [512, 512], [512, 511], [511, 512], ast=[1, 512]) == (1, 1, 1, 512, 512, 511, 0)
    assert mm_plan("bf16", [2, 2, 512, 512], [2, 2, 512, 512], [2, 2, 512, 512]) == (4, 0, 1, 512, 512, 512, 0)
    assert mm_plan("bf16", [4, 256, 512], [4, 256, 384], [4, 384, 512], which=1) == (4, 0, 0, 256, 384, 512, 0)
    assert mm_plan("bf16", [4, 256, 512], [4, 256, 384], [4, 384, 512], which=2) == (4, 1, 1, 384, 512, 256, 0)
    assert mm_plan("bf16", [256, 512], [256, 383], [383, 512], which=2) == (1, 1, 1, 383, 512, 256, 1)


def test_f32_products_of_short_reductions_stay_where_they_are_more_exact():
    """Below K = 192 the sums of the CUDA cores are closer to 64 bits than the split into two tf32 parts: ragged rows, rank 4 and
    batched backward products; the plain form keeps the split kernel at any K."""
    for k, taken in ((191, 0), (192, 1)):
        assert (mm_plan("f32", [1030, 515], [1030, k], [k, 515]) != 0) == taken
        assert (mm_plan("f32", [1030, 512], [1030, k], [k, 512], aoff=1) != 0) == taken
        assert (mm_plan("f32", [2, 4, 512, 512], [2, 4, 512, k // 4 * 4], [2, 4, k // 4 * 4, 512]) != 0) == taken
        assert (mm_plan("f32", [8, 512, k], [8, 512, 512], [8, 512, k], which=1) != 0) == taken
        assert (mm_plan("f32", [8, k, 512], [8, k, 512], [8, 512, 512], which=2) != 0) == taken
    assert mm_plan("f32", [1024, 512], [1024, 64], [64, 512])[0] == 1


def test_copies_stay_small_and_few_outputs_stay_with_their_kernel():
    # a vector is K-major whatever its strides say: nothing is copied where a [K, 1] matrix would grow eightfold
    assert mm_plan("bf16", [1, 1], [1, 1 << 24], [1 << 24, 1]) == (1, 0, 0, 1, 1, 1 << 24, 4)
    assert mm_plan("bf16", [1, 4096], [1, 4096], [4096, 4096], ast=[1, 1]) == (1, 0, 1, 1, 4096, 4096, 0)
    assert mm_plan("f32", [2048, 1], [2048, 16384], [16384, 1], ast=[1, 2048]) == (1, 1, 0, 2048, 1, 16384, 4)
    # rows of two elements: four times their size, taken while that is little memory
    assert mm_plan("bf16", [2, 4096], [2, 1 << 20], [1 << 20, 4096], ast=[1, 2])[6] == 1
    assert mm_plan("bf16", [2, 4096], [2, 1 << 22], [1 << 22, 4096], ast=[1, 2]) == 0
    assert mm_plan("f32", [70000, 40000], [70000, 32767], [32767, 40000]) == 0              # 9 GB of copies
    # at most 1024 outputs, 2048 terms or more
    assert mm_plan("bf16", [32, 32], [32, 4095], [4095, 32]) == 0
    assert mm_plan("bf16", [32, 32], [32, 4096], [4096, 32])[0] == 1
    assert mm_plan("bf16", [32, 32], [32, 4096], [4096, 32], bst=[1, 4096]) == 0
    assert mm_plan("bf16", [32, 32], [32, 8192], [8192, 32])[0] == 1
    assert mm_plan("bf16", [16, 64], [16, 2048], [2048, 64])[0] == 1                         # no copies
    assert mm_plan("bf16", [16, 63], [16, 2048], [2048, 63]) == 0
    assert mm_plan("bf16", [100, 10], [100, 4096], [4096, 10], ast=[1, 100])[0] == 1
    assert mm_plan("bf16", [100, 10], [100, 4095], [4095, 10], ast=[1, 100]) == 0
    assert mm_plan("bf16", [100, 10], [100, 4096], [4096, 10]) == 0
    assert mm_plan("f16", [8, 8], [8, 16384], [16384, 8]) == 0
    assert mm_plan("f16", [8, 8], [8, 32768], [32768, 8])[0] == 1
    assert mm_plan("bf16", [32, 32], [32, 16384], [16384, 32])[0] == 1                       # 2^24 multiply-adds, plain form: as ever
    assert mm_plan("f32", [5, 5], [5, 1 << 20], [1 << 20, 5]) == 0
    # f32: a block per output is more exact than the drained sums of the forms that are new to the tensor cores
    assert mm_plan("f32", [10, 100], [10, 60000], [60000, 100])[0] == 1
    assert mm_plan("f32", [10, 100], [10, 60000], [60000, 100], ast=[1, 10]) == 0
    assert mm_plan("f32", [20, 50], [20, 1 << 18], [1 << 18, 50]) == 0
    assert mm_plan("f32", [784, 1], [784, 65536], [65536, 1], ast=[1, 784]) == 0


def test_small_16_bit_products_with_long_reductions_take_the_tensor_core_kernel():
    assert mm_plan("bf16", [64, 64], [64, 256], [256, 64])[0] == 1
    assert mm_plan("bf16", [64, 64], [64, 255], [255, 64]) == 0        # fewer than 256 terms
    assert mm_plan("f16", [32, 32], [32, 256], [256, 32])[0] == 1      # 2^18 multiply-adds
    assert mm_plan("f16", [31, 32], [31, 256], [256, 32]) == 0
    assert mm_plan("f32", [64, 64], [64, 256], [256, 64]) == 0         # f32 keeps the element-type loop's order below 2^24


def test_f32_products_take_the_split_tf32_kernel_when_rows_are_16_byte_multiples():
    """f32: the contiguous extent of each matrix must be a multiple of 4 elements (16 bytes for TMA), not 8."""
    D = 8192
    assert mm_path([2, 2, 2, 2048, D, 2048, D, D, D, D, 1, 1, D, 0, 0], 2048 * D, f32=True) == (1, 0, 0, 2048, D, D)
    # conv forward at the benchmark shape: cols [200704, 2304] . weight^T view of [256, 2304]
    assert mm_path([2, 2, 2, 200704, 256, 200704, 2304, 2304, 256, 2304, 1, 1, 2304, 0, 0], 200704 * 256, f32=True) == (1, 0, 0, 200704, 256, 2304)
    assert mm_path([2, 2, 2, 512, 516, 512, 512, 512, 516, 512, 1, 516, 1, 0, 0], 512 * 516, f32=True)[0] == 1   # 516 = 4 * 129
    assert mm_path([2, 2, 2, 64, 64, 64, 64, 64, 64, 64, 1, 64, 1, 0, 0], 64 * 64, f32=True)[0] == 0             # small: SIMT, bit-exact order


def test_split_k_plan():
    """Few output tiles and a long reduction are cut along K so that every SM gets a tile; products that already fill
    the GPU, short reductions and K that does not divide are left alone."""
    lib = _lib.load()
    sk = lib.mx_debug_splitk_slices
    assert sk(18, 200704, 64, 148) == 8          # the conv weight gradient at the benchmark shape: 144 tiles on 148 SMs
    assert sk(36, 200704, 32, 148) == 4          # the same product in f32 (128 x 128 tiles)
    assert sk(4096, 8192, 64, 148) == 1          # the MLP products fill the GPU
    assert sk(4, 2048, 64, 148) == 1             # reduction too short to be worth a second pass
    assert sk(2, 65600, 64, 148) == 1 or 65600 % (64 * sk(2, 65600, 64, 148)) == 0
    for tiles, k in ((1, 1 << 20), (3, 65536), (10, 16384)):
        s_ = sk(tiles, k, 64, 148)
        assert s_ >= 1 and (k // 64) % s_ == 0 and k // s_ >= 1024


def test_b_panel_resident_schedule_is_for_short_reductions_with_many_row_tiles():
    lib = _lib.load()
    keep = lib.mx_debug_gemm_keep_b_ctas
    assert keep(1568, 9, 4, 1, 148) == 16      # the conv input-gradient product (200704 x 2304 x 256): 16 CTAs per column tile
    assert keep(1568, 9, 5, 1, 148) == 0       # K = 320 does not fit the four-slot ring
    assert keep(1568, 9, 4, 2, 148) == 0       # batched products keep the general schedule
    assert keep(40, 9, 4, 1, 148) == 0         # too few row tiles per CTA to spread the panel's load over
    assert keep(1568, 200, 4, 1, 148) == 0     # more column tiles than CTAs
    assert keep(400, 1, 2, 1, 148) == 0        # 148 CTAs on one column tile: fewer than four row tiles each
    assert keep(1000, 1, 2, 1, 148) == 148
