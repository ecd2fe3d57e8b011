"""The native form of device.dispatch hands an op the same arguments as ctypes does, and leaves to the interpreted form what it does not take."""
import ctypes

import pytest

from maidenx_b200 import _signatures as sig
from maidenx_b200 import dtypes as D

native = pytest.importorskip("maidenx_b200._dispatch")
FAMILIES = ["binary", "binary_inplace", "unary_const", "reduce", "matmul", "matmul_backward", "conv", "pad_const"]
BLOCK = (ctypes.c_size_t * 64)()


@pytest.fixture
def seen():
    """The module bound to calls that record what arrives; bound to the library again afterwards."""
    from maidenx_b200 import device
    got = {"general": [], "ops": []}

    def begin(dev, words, count, block):
        got["begin"] = (dev, [words[i] for i in range(count)])
        ctypes.memmove(BLOCK, words, 8 * count)
        block[0] = ctypes.addressof(BLOCK)
        return 7 if dev == 9 else 0

    def end(block):
        got["end"] = block
        return got.get("status", 0)

    c_begin = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_size_t), ctypes.c_size_t, ctypes.POINTER(ctypes.c_void_p))(begin)
    c_end = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p)(end)
    address = lambda f: ctypes.cast(f, ctypes.c_void_p).value  # noqa: E731
    native.bind(address(c_begin), address(c_end))
    got["keep"] = [c_begin, c_end]
    native.setup(lambda *a, **k: got["general"].append((a, k)), lambda *a: None, lambda *a: ("begin failed", a), lambda *a: ("op failed", a))
    yield got
    native.setup(device._dispatch_general, device._register, device._check, device._raise_last_error)
    try:
        from maidenx_b200 import _lib
        lib = _lib.load()
        native.bind(address(lib.mx_dispatch_begin), address(lib.mx_dispatch_end))
    except Exception:
        pass


def _fake(got, family, d):
    """An op of the family that records its arguments; returns its name and its ctypes signature."""
    types = sig.argtypes(family, d)
    fn = ctypes.CFUNCTYPE(None, *types)(lambda *a: got["ops"].append(a))
    got["keep"].append(fn)
    at = {"unary_const": 4, "pad_const": 6}.get(family)
    letters = "".join("P" if t is ctypes.c_void_p else "S" if t is ctypes.c_size_t and i != at else t._type_ for i, t in enumerate(types))
    if at is not None:
        letters = letters[:at] + types[at]._type_ + letters[at + 1:]
    name = f"fake_{family}"
    assert native.register(name, d.name, ctypes.cast(fn, ctypes.c_void_p).value, letters, letters.index("P"))
    return name, types, at


@pytest.mark.parametrize("family,d", [(f, D.F32) for f in FAMILIES] + [(f, d) for f in ("unary_const", "pad_const") for d in D.ALL if d is not D.F32],
                         ids=lambda v: v if isinstance(v, str) else v.name)
def test_arguments_arrive_as_ctypes_converts_them(seen, family, d):
    name, types, at = _fake(seen, family, d)
    scalars = [-2.5, 3] if d.name in ("f32", "f64") else [0, 1, 2, 255, -1, 1 << 40, True] if d.name == "bool" else [0, 3, -1, (1 << 64) + 5]
    meta = types.index(ctypes.c_void_p)
    for s in scalars if at is not None else [None]:
        plain = [s if i == at else "META" if i == meta else 1000 + i if t is ctypes.c_size_t else (1 << 63) + i for i, t in enumerate(types)]
        last = max(i for i, t in enumerate(types) if t is ctypes.c_void_p)
        plain[last] = None
        seen["ops"].clear()
        native.dispatch(name, d.name, [5, 1, 2**64 - 1], *plain, device=3)
        if d.name == "bool" and s is True or type(s) in (int, float, type(None)):
            assert not seen["general"] and seen["begin"] == (3, [5, 1, 2**64 - 1]) and seen["end"] == ctypes.addressof(BLOCK)
        want = [t(v).value for t, v in zip(types, [ctypes.addressof(BLOCK) if v == "META" else v for v in plain])]
        assert list(seen["ops"][0]) == want


def test_other_calls_go_to_the_interpreted_form(seen):
    name, _, _ = _fake(seen, "unary_const", D.F16)
    good = (name, "f16", [1, 1, 0], 1, 1, "META", 16, 3, 32)
    other = [
        ((name, "f16", (1, 1, 0), 1, 1, "META", 16, 3, 32), {}), ((name, "f16", [], 1, 1, "META", 16, 3, 32), {}), ((name, "f16", None, 1, 1, "META", 16, 3, 32), {}),
        ((name, "f16", [1, -1, 0], 1, 1, "META", 16, 3, 32), {}), ((name, "f16", [1, 1.0, 0], 1, 1, "META", 16, 3, 32), {}), ((name, "f16", [1] * 65, 1, 1, "META", 16, 3, 32), {}),
        ((name, "f16", [1, 1, 0], ctypes.c_size_t(1), 1, "META", 16, 3, 32), {}), ((name, "f16", [1, 1, 0], 1, 1, "META", 16, 2.0, 32), {}),
        ((name, "f16", [1, 1, 0], 1, None, "META", 16, 3, 32), {}), ((name, "f16", [1, 1, 0], 1, 1, 8, 16, 3, 32), {}), ((name, "f16", [1, 1, 0], 1, 1, "META", 16, 3), {}),
        (good + (1,), {}), (good, {"metadata_on_host": True}), (good, {"check": 1}), (good[:2], {}),
    ]
    for n, (args, kw) in enumerate(other):
        native.dispatch(*args, **kw)
        assert len(seen["general"]) == n + 1 and seen["general"][-1] == (args, kw) and not seen["ops"], n
    assert native.dispatch(*good, device=9) == ("begin failed", (7, "metadata upload")) and not seen["ops"]
    seen["status"] = 3
    assert native.dispatch(*good) == ("op failed", (name, "f16")) and native.dispatch(*good, check=False) is None
