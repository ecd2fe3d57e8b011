"""Parity of conv2d im2col / col2im against the CPU oracle, through the C ABI, on a B200.
Both are copies or short fixed-order sums in the element type, so the bar is bit-exact for
all four float dtypes.  Nothing in the reference pins these values (its Conv2d tests check
shapes only), so the oracle's restatement of crates/maidenx_cpu/src/nn/conv.rs is the
definition.  col2im is exercised both with num_els = the full col length and with the value
the reference's Conv2d passes, B*C*H*W (crates/maidenx_nn/src/layers/conv.rs:393), which
makes every col entry at or beyond it invisible.
"""
import numpy as np
import pytest

import harness as H
from maidenx_b200 import dtypes as D

pytestmark = pytest.mark.gpu


def cases():
    """(name, B, C, H, W, kh, kw, ph, pw, sh, sw)"""
    return [
        ("3x3-s1-p1", 2, 3, 8, 8, 3, 3, 1, 1, 1, 1),
        ("3x3-s1-p1-vec", 2, 4, 16, 16, 3, 3, 1, 1, 1, 1),
        ("5x5-s2-p2", 1, 2, 13, 11, 5, 5, 2, 2, 2, 2),
        ("2x3-mixed", 2, 2, 9, 10, 2, 3, 0, 1, 1, 2),
        ("1x1", 3, 5, 7, 7, 1, 1, 0, 0, 1, 1),
        ("no-pad", 1, 3, 12, 12, 3, 3, 0, 0, 1, 1),
        ("s3", 1, 1, 20, 17, 3, 3, 1, 1, 3, 3),
        ("big-plane", 1, 2, 56, 56, 3, 3, 1, 1, 1, 1),
        # stride-1 vector fast paths: widths that are multiples of the 16-byte vector, kw in {1,3,5,7}
        ("5x5-s1-p2-vec", 2, 2, 16, 24, 5, 5, 2, 2, 1, 1),
        ("7x7-s1-p3-vec", 1, 1, 16, 16, 7, 7, 3, 3, 1, 1),
        ("1x1-vec", 2, 3, 8, 16, 1, 1, 0, 0, 1, 1),
        ("1x3-vec", 1, 2, 9, 16, 1, 3, 0, 1, 1, 1),
        ("3x1-vec", 1, 2, 9, 16, 3, 1, 1, 0, 1, 1),
        ("3x3-s1-p0", 1, 2, 10, 10, 3, 3, 0, 0, 1, 1),
        ("3x3-s1-p1-tall", 3, 2, 40, 8, 3, 3, 1, 1, 1, 1),
    ]


def _geom(c):
    _, B, C, Hh, W, kh, kw, ph, pw, sh, sw = c
    oh = (Hh + 2 * ph - kh) // sh + 1
    ow = (W + 2 * pw - kw) // sw + 1
    return B, C, Hh, W, kh, kw, oh, ow, ph, pw, sh, sw


@pytest.mark.parametrize("dt", D.FLOATS, ids=lambda d: d.name)
def test_im2col(oracle, cuda, dt):
    rng = np.random.default_rng(31)
    for c in cases():
        B, C, Hh, W, kh, kw, oh, ow, ph, pw, sh, sw = _geom(c)
        meta = H.conv_metadata(B, C, Hh, W, kh, kw, oh, ow, ph, pw, sh, sw)
        x = H.random_store(rng, dt, B * C * Hh * W, dist="normal")
        n = B * C * kh * kw * oh * ow
        ref = H.run_im2col(oracle, dt, meta, n, x)
        got = H.run_im2col(cuda, dt, meta, n, x)
        H.assert_same("conv2d_im2col", dt, got, ref, what=c[0])


@pytest.mark.parametrize("dt", D.FLOATS, ids=lambda d: d.name)
def test_col2im(oracle, cuda, dt):
    rng = np.random.default_rng(32)
    for c in cases():
        B, C, Hh, W, kh, kw, oh, ow, ph, pw, sh, sw = _geom(c)
        meta = H.conv_metadata(B, C, Hh, W, kh, kw, oh, ow, ph, pw, sh, sw)
        ncol = B * C * kh * kw * oh * ow
        col = H.random_store(rng, dt, ncol, dist="normal")
        out_len = B * C * Hh * W
        for num_els in (ncol, min(ncol, out_len)):
            ref = H.run_col2im(oracle, dt, meta, num_els, col, out_len)
            got = H.run_col2im(cuda, dt, meta, num_els, col, out_len)
            H.assert_same("conv2d_col2im", dt, got, ref, what=f"{c[0]} num_els={num_els}")


def test_im2col_col2im_adjoint(cuda):
    """<im2col(x), y> == <x, col2im(y)> (the two are adjoint linear maps): a size-independent
    property, checked here in f64."""
    rng = np.random.default_rng(33)
    dt = D.F64
    B, C, Hh, W, kh, kw, oh, ow, ph, pw, sh, sw = _geom(("", 2, 3, 10, 9, 3, 3, 1, 1, 2, 1))
    meta = H.conv_metadata(B, C, Hh, W, kh, kw, oh, ow, ph, pw, sh, sw)
    ncol = B * C * kh * kw * oh * ow
    x = rng.standard_normal(B * C * Hh * W)
    y = rng.standard_normal(ncol)
    cx = H.run_im2col(cuda, dt, meta, ncol, x)
    ty = H.run_col2im(cuda, dt, meta, ncol, y, x.size)
    assert np.isclose(np.dot(cx, y), np.dot(x, ty), rtol=1e-12)


MANY_PLANES = [
    # name, B, C, H, W, kh, kw, ph, pw, sh, sw: enough planes for several per block, maps that are whole vectors and maps that are not
    ("14x14", 7, 131, 14, 14, 3, 3, 1, 1, 1, 1),
    ("7x7-s2", 5, 211, 7, 7, 3, 3, 1, 1, 2, 2),
    ("7x7-s2-groups", 120, 293, 7, 7, 3, 3, 1, 1, 2, 2),  # 29 planes a block, in groups of 7 (f32) or 14 (16-bit types), the last one cut short
    ("9x11-5x5", 3, 300, 9, 11, 5, 5, 2, 2, 1, 1),
    ("1x1-odd", 4, 401, 5, 5, 1, 1, 0, 0, 1, 1),
    ("17x19", 4, 200, 17, 19, 3, 3, 1, 1, 1, 1),      # more pixels than a block has threads, blocks enough
    ("7x7", 12, 300, 7, 7, 3, 3, 1, 1, 1, 1),
    ("15x15-few", 1, 9, 15, 15, 3, 3, 1, 1, 1, 1),    # too few planes to share blocks
    ("large-planes-few-outputs", 2, 3, 150, 150, 15, 15, 0, 0, 15, 15),
    ("large-planes", 1, 3, 160, 160, 3, 3, 1, 1, 2, 2),
    ("even-kernel", 3, 257, 6, 10, 2, 4, 1, 0, 1, 3),
    ("one-output-row", 9, 120, 7, 31, 7, 7, 0, 0, 1, 1),   # square kernels by ranges: most of a pixel's terms lie outside
    ("a-quarter-of-the-terms", 9, 120, 12, 12, 7, 7, 0, 0, 1, 1),
    ("half-of-the-terms", 9, 120, 14, 14, 5, 5, 0, 0, 1, 1),
    ("plane-beyond-shared-memory", 1, 2, 170, 331, 3, 3, 1, 1, 2, 2),
]


@pytest.mark.parametrize("dt", D.FLOATS, ids=lambda d: d.name)
@pytest.mark.parametrize("case", MANY_PLANES, ids=lambda c: c[0])
def test_planes_sharing_a_block(oracle, cuda, dt, case):
    """Bit-exact like every case of this file; also column buffers that end inside a plane (num_els)."""
    rng = np.random.default_rng(34)
    B, C, Hh, W, kh, kw, oh, ow, ph, pw, sh, sw = _geom(case)
    meta = H.conv_metadata(B, C, Hh, W, kh, kw, oh, ow, ph, pw, sh, sw)
    ncol, out_len = B * C * kh * kw * oh * ow, B * C * Hh * W
    x, col = H.random_store(rng, dt, out_len, dist="normal"), H.random_store(rng, dt, ncol, dist="normal")
    for n in (ncol, ncol - kh * kw * oh * ow // 2 - 1):
        H.assert_same("conv2d_im2col", dt, H.run_im2col(cuda, dt, meta, n, x), H.run_im2col(oracle, dt, meta, n, x), what=f"{case[0]} {n}")
    for n in (ncol, ncol // 2 + 1):
        H.assert_same("conv2d_col2im", dt, H.run_col2im(cuda, dt, meta, n, col, out_len), H.run_col2im(oracle, dt, meta, n, col, out_len), what=f"{case[0]} {n}")


def test_threads_with_planes_of_different_sizes(cuda):
    """Threads whose planes need different amounts of shared memory beyond 48 KB, calling as fast as they can: none may take back the
    limit that another has just asked for (its launch would be refused)."""
    import ctypes
    import threading

    from maidenx_b200 import _lib

    dt, lib, op = D.F32, _lib.load(), _lib.op("conv2d_im2col", "f32")
    start, trouble = threading.Barrier(4), []

    def work(side):
        C, o = 2, (side + 2 - 3) // 2 + 1
        meta = np.asarray(H.conv_metadata(1, C, side, side, 3, 3, o, o, 1, 1, 2, 2), dtype=np.uint64)
        x = H.random_store(np.random.default_rng(side), dt, C * side * side, dist="normal")
        n = C * 9 * o * o
        bx, bc = cuda.dev.CudaBuffer.from_host(x), cuda.dev.CudaBuffer.from_host(np.zeros(n, np.float32))
        start.wait()
        for _ in range(4000):
            op(ctypes.c_size_t(n), meta.ctypes.data, bx.ptr, bc.ptr)
        trouble.append(lib.mx_last_error())
        lib.mx_clear_error()
        cuda.dev.synchronize()
        trouble.append(0 if np.array_equal(bc.to_host(np.float32, n), H.run_im2col(cuda, dt, list(map(int, meta)), n, x)) else side)
        bx.free()
        bc.free()

    ts = [threading.Thread(target=work, args=(side,)) for side in (121, 213, 151, 187)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert trouble == [0] * 8


@pytest.mark.parametrize("dt", D.FLOATS, ids=lambda d: d.name)
@pytest.mark.parametrize("case", [(3, 5, 0, 6, 1, 3, 1, 1), (2, 7, 6, 0, 3, 1, 1, 2), (1, 1, 0, 0, 2, 2, 1, 1), (40, 60, 0, 1, 1, 1, 1, 0)], ids=str)
def test_images_of_no_pixels(cuda, dt, case):
    """H or W of zero: padding alone gives output positions, and every column entry is a zero of it."""
    B, C, Hh, W, kh, kw, ph, pw = case
    oh, ow = Hh + 2 * ph - kh + 1, W + 2 * pw - kw + 1
    meta = H.conv_metadata(B, C, Hh, W, kh, kw, oh, ow, ph, pw, 1, 1)
    n = B * C * kh * kw * oh * ow
    assert n > 0
    got = H.run_im2col(cuda, dt, meta, n, H.random_store(np.random.default_rng(1), dt, 1, dist="normal"))
    assert np.array_equal(D.decode(got, dt), np.zeros(n))


GROUPS = [
    # several groups of planes a block, the last block and the last group incomplete; groups of one, two and four planes; kernels of 3, 5, 7 (terms at fixed distances) and others
    ("14x14-3", 9, 277, 14, 14, 3, 3, 1, 1, 1, 1), ("13x13-5", 8, 313, 13, 13, 5, 5, 2, 2, 1, 1), ("7x7-7", 11, 223, 7, 7, 7, 7, 3, 3, 1, 1), ("6x10-3-nopad", 10, 251, 6, 10, 3, 3, 0, 0, 1, 1),
    ("9x9-7-wide-pad", 7, 350, 9, 9, 7, 7, 5, 4, 1, 1), ("8x9-3x5", 6, 401, 8, 9, 3, 5, 1, 2, 1, 1), ("11x7-3-s2", 9, 301, 11, 7, 3, 3, 1, 1, 2, 2), ("4x4-5", 3, 797, 4, 4, 5, 5, 2, 2, 1, 1),
]


@pytest.mark.parametrize("dt", D.FLOATS, ids=lambda d: d.name)
@pytest.mark.parametrize("case", GROUPS, ids=lambda c: c[0])
def test_groups_of_planes_in_a_block(oracle, cuda, dt, case):
    test_planes_sharing_a_block(oracle, cuda, dt, case)
