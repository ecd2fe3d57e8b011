"""The metadata blocks of mx_dispatch_begin / mx_dispatch_end: slots the launcher reads where they lie, and device blocks for what does not fit."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _begin(lib, words):
    block = ctypes.c_void_p()
    raw = np.asarray(words, dtype=np.uint64).tobytes()
    assert lib.mx_dispatch_begin(0, raw, len(words), ctypes.byref(block)) == 0 and block.value
    return block


def test_blocks_open_at_once_read_back_and_given_back(cuda):
    from maidenx_b200 import _lib, device
    lib = _lib.load()
    neg = _lib.op("neg", "f32")
    x = np.arange(1, 401, dtype=np.float32)
    src, dst = device.CudaBuffer.from_host(x), device.CudaBuffer(4 * 400)
    try:
        blocks = [_begin(lib, [n + 1, 1, 0]) for n in range(300)]        # more than there are slots
        assert len({b.value for b in blocks}) == 300
        for n, b in enumerate(blocks):
            back = np.zeros(3, dtype=np.uint64)
            assert lib.cuda_memcpy_d2h(back.ctypes.data, b, 24) == 0 and list(back) == [n + 1, 1, 0]
            dst.fill_from(np.zeros(400, np.float32))
            neg(n + 1, 1, b, src.ptr, dst.ptr)
            got = dst.to_host(np.float32, 400)
            assert np.array_equal(got[:n + 1], -x[:n + 1]) and not got[n + 1:].any()
        assert lib.cuda_free(blocks.pop()) == 0                          # the call that mx_dispatch_end makes
        assert all(lib.mx_dispatch_end(b) == 0 for b in blocks)
        b = _begin(lib, [2, 3, 100, 1, 0])                               # dims [2, 3]
        new = np.array([3, 2, 1, 3, 0], dtype=np.uint64)                 # the transposed view, written over it
        assert lib.cuda_memcpy_h2d(b, new.ctypes.data, 40) == 0
        neg(6, 2, b, src.ptr, dst.ptr)
        assert np.array_equal(dst.to_host(np.float32, 6), -x[:6].reshape(2, 3).T.reshape(-1)) and lib.mx_dispatch_end(b) == 0
        long = _begin(lib, [1] * 300 + [4] + [1] * 300 + [1, 0])         # beyond a slot: a device block, refused for its rank
        neg(4, 301, long, src.ptr, dst.ptr)
        assert lib.mx_dispatch_end(long) == 2
        lib.mx_clear_error()
        short = _begin(lib, [4])                                         # fewer words than the op reads
        neg(4, 1, short, src.ptr, dst.ptr)
        assert lib.mx_dispatch_end(short) == 2
    finally:
        lib.mx_clear_error()
        src.free()
        dst.free()


def test_words_of_a_block_written_anew(cuda):
    """A block may be written in part, and past the words it was given, from the host or the device, with work queued on the stream: the next op reads what was
    written, and a block that is handed out again holds nothing of it."""
    from maidenx_b200 import _lib, device
    lib = _lib.load()
    neg, x = _lib.op("neg", "f32"), np.arange(1, 1 << 25, dtype=np.float32)
    src, dst, busy = device.CudaBuffer.from_host(x), device.CudaBuffer(4 * 16), device.CudaBuffer(4 * x.size)
    try:
        def words(*v):
            return np.array(v, dtype=np.uint64)

        for i in range(100):
            block = _begin(lib, [4, 1, 0])
            for _ in range(3):  # the device is busy when the words arrive
                neg(x.size, 1, None, src.ptr, busy.ptr)
            offset = words(3 * i)
            if i % 2:
                on_device = device.CudaBuffer.from_host(offset)
                assert lib.cuda_memcpy_d2d(block.value + 16, on_device.ptr, 8) == 0
                on_device.free()
            else:
                assert lib.cuda_memcpy_h2d(block.value + 16, offset.ctypes.data, 8) == 0
            neg(4, 1, block, src.ptr, dst.ptr)
            assert lib.mx_dispatch_end(block) == 0
            assert np.array_equal(dst.to_host(np.float32, 4), -x[3 * i:3 * i + 4]), i
        table = lib.mx_metadata_table_size()
        block = _begin(lib, [4])                                          # fewer words than the op reads, completed afterwards
        rest = words(1, 7)
        assert lib.cuda_memcpy_h2d(block.value + 8, rest.ctypes.data, 16) == 0
        neg(4, 1, block, src.ptr, dst.ptr)
        assert lib.mx_last_error() == 0 and np.array_equal(dst.to_host(np.float32, 4), -x[7:11])
        copy = device.CudaBuffer(24)
        assert lib.cuda_memcpy_d2d(copy.ptr, block, 24) == 0 and lib.mx_dispatch_end(block) == 0
        block = _begin(lib, [9, 9, 9])
        assert list(copy.to_host(np.uint64, 3)) == [4, 1, 7] and lib.mx_dispatch_end(block) == 0
        copy.free()
        assert lib.mx_metadata_table_size() == table                      # nothing is remembered for addresses inside a slot
        block = _begin(lib, [9])
        neg(4, 1, block, src.ptr, dst.ptr)                                # the words of its last use do not count
        assert lib.mx_dispatch_end(block) == 2
        block, long = _begin(lib, [4, 1, 0]), np.zeros(300, np.uint64)
        assert lib.cuda_memcpy_h2d(block.value, long.ctypes.data, 2400) != 0  # past the end of the slot: refused, nothing written
    finally:
        lib.mx_clear_error()
        for b in (src, dst, busy):
            b.free()
    assert lib.mx_dispatch_end(block) == 0


def test_threads_share_the_slots(cuda):
    from maidenx_b200 import device
    bad = []

    def work(seed):
        n = 100 + seed
        x = np.arange(n, dtype=np.float32) + seed
        a, o = device.CudaBuffer.from_host(x), device.CudaBuffer(4 * n)
        for _ in range(300):
            device.dispatch("neg", "f32", [n, 1, 0], n, 1, "META", a.ptr, o.ptr)
        if not np.array_equal(o.to_host(np.float32, n), -x):
            bad.append(seed)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(6)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad


@pytest.mark.parametrize("n", [1, 1000, 300000, 3000001])
def test_each_launch_of_a_chain_sees_the_one_before(cuda, n):
    """Kernels are scheduled when the one before them ends: a chain in which every launch reads what the last one wrote, of sums (whose last block folds the others'
    parts), passes over vectors and small ones after large ones.  Whole numbers below 2^24: exact."""
    from maidenx_b200 import device
    x = np.arange(n, dtype=np.float32) % 5
    a, b, s = device.CudaBuffer.from_host(x), device.CudaBuffer(4 * n), device.CudaBuffer.from_host(np.zeros(1, np.float32))
    total = 0.0
    try:
        for _ in range(20):
            device.dispatch("neg", "f32", [n, 1, 0], n, 1, "META", a.ptr, b.ptr)
            device.dispatch("sub", "f32", [n, 1, 1, 0, 0], n, 1, "META", a.ptr, b.ptr, a.ptr)          # a = 2 a
            device.dispatch("neg", "f32", [n, 1, 0], n, 1, "META", b.ptr, b.ptr)                        # b = the a before
            device.dispatch("sub", "f32", [n, 1, 1, 0, 0], n, 1, "META", a.ptr, b.ptr, a.ptr)          # a as it was
            device.dispatch("sum_to_shape", "f32", [n, 1, 1, 0], n, 1, "META", a.ptr, s.ptr)
        total = float(s.to_host(np.float32, 1)[0])
        assert total == x.sum(dtype=np.float64) and np.array_equal(a.to_host(np.float32, n), x)
    finally:
        for buf in (a, b, s):
            buf.free()


READERS = {  # name: elements read, elements written, words and arguments of the call (x: what it reads, out: what it writes)
    "softmax_rows": (2048 * 1024, 2048 * 1024, lambda x, out: ("softmax", [2048, 1024, 1024, 1, 0], 2048 * 1024, 2, 1, "META", x, out)),
    "softmax_rows_of_a_block": (256 * 8192, 256 * 8192, lambda x, out: ("softmax", [256, 8192, 8192, 1, 0], 256 * 8192, 2, 1, "META", x, out)),
    "softmax_ragged": (2047 * 197, 2047 * 197, lambda x, out: ("softmax", [2047, 197, 197, 1, 0], 2047 * 197, 2, 1, "META", x, out)),
    "softmax_columns": (512 * 1024, 512 * 1024, lambda x, out: ("softmax", [512, 1024, 1024, 1, 0], 512 * 1024, 2, 0, "META", x, out)),
    "product": (1024 * 512, 1024 * 1024, lambda x, out: ("matmul", [2, 2, 2, 1024, 1024, 1024, 512, 512, 1024, 512, 1, 1, 512, 0, 0], 1024 * 1024, "META", x, x, out)),
    "im2col": (16 * 32 * 28 * 28, 16 * 32 * 9 * 28 * 28, lambda x, out: ("conv2d_im2col", [16, 32, 28, 28, 3, 3, 28, 28, 1, 1, 1, 1], 16 * 32 * 9 * 28 * 28, "META", x, out)),
    "col2im": (16 * 32 * 9 * 28 * 28, 16 * 32 * 28 * 28, lambda x, out: ("conv2d_col2im", [16, 32, 28, 28, 3, 3, 28, 28, 1, 1, 1, 1], 16 * 32 * 9 * 28 * 28, "META", x, out)),
}


@pytest.mark.parametrize("dt", ["f32", "bf16"])
@pytest.mark.parametrize("name", READERS)
def test_readers_see_what_the_launch_before_them_wrote(cuda, name, dt):
    """An op that reads, right behind it, the whole buffer that a pass over vectors has just written, twenty times with other values each time: bit for bit what it
    gives with the device idle in between.  A load ahead of the kernel's wait would find the values of the time before."""
    from maidenx_b200 import _lib, device, dtypes as D
    lib = _lib.load()
    t = D.BY_NAME[dt]
    n_in, n_out, call = READERS[name]
    rng = np.random.default_rng(n_in)
    bufs = [device.CudaBuffer.from_host(D.encode(rng.standard_normal(n_in).astype(np.float32), t)) for _ in range(3)]
    x = device.CudaBuffer.from_host(np.zeros(n_in, t.np_storage))
    outs = [[device.CudaBuffer.from_host(np.zeros(n_out, t.np_storage)) for _ in range(3)] for _ in range(2)]
    try:
        for idle in (True, False):
            for i in range(20):
                device.dispatch("neg", dt, [n_in, 1, 0], n_in, 1, "META", bufs[i % 3].ptr, x.ptr)
                if idle:
                    assert lib.mx_device_synchronize() == 0
                op, *args = call(x.ptr, outs[idle][i % 3].ptr)
                device.dispatch(op, dt, *args)
        for i in range(3):
            a, b = (outs[k][i].to_host(t.np_storage, n_out) for k in range(2))
            assert a.any() and np.array_equal(a, b)
    finally:
        for b in [x, *bufs, *outs[0], *outs[1]]:
            b.free()
