"""Device memory and the reference-style dispatch pattern, through the library's own wrappers.

`CudaBuffer` mirrors the reference's buffer type (crates/maidenx_core/src/buffer/cuda.rs:21-40,
58-75): `cuda_malloc` on creation, `cuda_free` on release, base pointer handed to the ops,
element offsets travelling in the metadata.  `dispatch` mirrors what every generated
function of crates/maidenx_core/src/be/ops/*.rs does around an op call: select the device,
provide the metadata block (mx_dispatch_begin: a slot of pinned memory, or cuda_malloc +
cuda_memcpy_h2d), call `cuda_<op>_<dtype>`, give the block back.
"""
from __future__ import annotations

import ctypes
import struct

import numpy as np

from . import _lib


class CudaError(RuntimeError):
    pass


def _check(code: int, what: str):
    if code != 0:
        lib = _lib.load()
        raise CudaError(f"{what}: {lib.cuda_error_string(code).decode()} ({code})")


class CudaBuffer:
    def __init__(self, nbytes: int):
        lib = _lib.load()
        self.nbytes = int(nbytes)
        p = ctypes.c_void_p()
        _check(lib.cuda_malloc(ctypes.byref(p), max(self.nbytes, 1)), "cuda_malloc")
        self.ptr = p.value

    @classmethod
    def from_host(cls, arr: np.ndarray) -> "CudaBuffer":
        arr = np.ascontiguousarray(arr)
        buf = cls(arr.nbytes)
        if arr.nbytes:
            _check(_lib.load().cuda_memcpy_h2d(buf.ptr, arr.ctypes.data, arr.nbytes), "cuda_memcpy_h2d")
        return buf

    def to_host(self, np_dtype, count: int) -> np.ndarray:
        out = np.empty(count, dtype=np_dtype)
        if out.nbytes:
            _check(_lib.load().cuda_memcpy_d2h(out.ctypes.data, self.ptr, out.nbytes), "cuda_memcpy_d2h")
        return out

    def fill_from(self, arr: np.ndarray):
        arr = np.ascontiguousarray(arr)
        assert arr.nbytes <= self.nbytes
        _check(_lib.load().cuda_memcpy_h2d(self.ptr, arr.ctypes.data, arr.nbytes), "cuda_memcpy_h2d")

    def free(self):
        if self.ptr:
            _lib.load().cuda_free(self.ptr)
            self.ptr = None

    def __del__(self):  # pragma: no cover
        try:
            self.free()
        except Exception:
            pass


def alloc_and_copy_dims(metadata) -> CudaBuffer:
    """crates/maidenx_cuda/src/lib.rs:177-193."""
    return CudaBuffer.from_host(np.asarray(metadata, dtype=np.uint64))


def last_error() -> str | None:
    lib = _lib.load()
    st = lib.mx_last_error()
    if st == 0:
        return None
    msg = f"status {st} at {lib.mx_last_error_where().decode()}"
    if st == 1:
        msg += f": {lib.cuda_error_string(lib.mx_last_cuda_error()).decode()}"
    return msg


def _raise_last_error(op: str, dtype_name: str):
    err = last_error()
    _lib.load().mx_clear_error()
    raise CudaError(f"cuda_{op}_{dtype_name}: {err}")


_packers = {}  # words of a metadata block -> packing function


def _dispatch_general(op: str, dtype_name: str, metadata, *args, device: int = 0, metadata_on_host: bool = False, check: bool = True):
    """`dispatch` with any arguments that ctypes and numpy take; the usual call is csrc/pydispatch.cpp's."""
    lib = _lib.load()
    if not metadata_on_host and type(metadata) is list and metadata:
        # packing with struct and two native calls around the op, whose metadata block is read where it is written
        pack = _packers.get(len(metadata))
        if pack is None:
            pack = _packers[len(metadata)] = struct.Struct(f"{len(metadata)}Q").pack
        try:
            words = pack(*metadata)
        except struct.error:
            words = None  # not whole 64-bit numbers: numpy's conversion below decides
        if words is not None:
            fn = _lib.op(op, dtype_name)
            block = ctypes.c_void_p()
            status = lib.mx_dispatch_begin(device, words, len(metadata), ctypes.byref(block))
            if status:
                _check(status, "metadata upload")
            try:
                fn(*[block if type(a) is str and a == "META" else a for a in args])
            finally:
                status = lib.mx_dispatch_end(block)
            if check and status:
                _raise_last_error(op, dtype_name)
            return
    _check(lib.cuda_set_device(device), "cuda_set_device")
    fn = _lib.op(op, dtype_name)
    mbuf = None
    keep = None
    if metadata is None:
        mptr = None
    elif metadata_on_host:
        keep = np.asarray(metadata, dtype=np.uint64)
        mptr = keep.ctypes.data
    else:
        mbuf = alloc_and_copy_dims(metadata)
        mptr = mbuf.ptr
    call_args = [mptr if (isinstance(a, str) and a == "META") else a for a in args]
    fn(*call_args)
    if mbuf is not None:
        mbuf.free()
    if check and lib.mx_last_error():
        _raise_last_error(op, dtype_name)


def _register(op: str, dtype_name: str):
    """Makes an entry point known to the native dispatch; raises where there is none."""
    lib = _lib.load()
    fn = _lib.op(op, dtype_name)
    address = lambda f: ctypes.cast(f, ctypes.c_void_p).value  # noqa: E731
    _native.bind(address(lib.mx_dispatch_begin), address(lib.mx_dispatch_end))
    types = "".join("P" if t is ctypes.c_void_p else "S" if t is ctypes.c_size_t else t._type_ for t in fn.argtypes)
    # the first pointer is the metadata block, by-value u64 scalars (the same C type as sizes) stand where the family says
    family, _ = _lib._ops.family[(op, dtype_name)]
    at = {"unary_const": 4, "unary_const_bool": 4, "pad_const": 6}.get(family)
    if at is not None:
        types = types[:at] + fn.argtypes[at]._type_ + types[at + 1:]
    _native.register(op, dtype_name, address(fn), types, types.index("P"))


try:
    from . import _dispatch as _native
except ImportError:  # not built: the interpreted form does the same
    dispatch = _dispatch_general
else:
    _native.setup(_dispatch_general, _register, _check, _raise_last_error)
    dispatch = _native.dispatch


def synchronize():
    _check(_lib.load().mx_device_synchronize(), "cudaDeviceSynchronize")
