"""Conv2d as a whole: im2col + matmul forward, matmul + col2im / matmul / sums backward.

CPU (no GPU needed): the oracle, composed op by op in the consistent ("direct") way, is a convolution — checked
against an independent float64 convolution, which is a second, formulation-independent pin of the oracle's
im2col / col2im (the reference's own tests only check Conv2d shapes, crates/maidenx_nn/src/layers/conv.rs:422-471).
GPU: the library's composition (mx_conv2d_forward / backward through the C ABI) against the oracle composed with
the same calls, for the literal reference call sequence (mode 0) and the direct one (mode 1), and mode 1 against
the float64 convolution.  Tolerances: f32 1e-4 and bf16 / f16 2e-2 of max(|ref|, sqrt(terms)).
"""
import numpy as np
import pytest

import conv2d_compose as CC
import harness as H
from maidenx_b200 import dtypes as D

# B, C, H, W, Cout, kh, kw, sh, sw, ph, pw
SMALL = [
    (2, 3, 8, 8, 4, 3, 3, 1, 1, 1, 1),
    (3, 2, 7, 9, 5, 3, 2, 2, 1, 1, 0),
    (1, 4, 6, 6, 3, 1, 1, 1, 1, 0, 0),
]
# the literal reference call sequence swaps the stride and padding slots, so the kernels see stride = padding:
# a zero padding would be a zero stride (a division by zero in the reference's own CPU backend)
LITERAL = [
    (2, 3, 8, 8, 4, 3, 3, 1, 1, 1, 1),
    (2, 3, 9, 8, 4, 3, 3, 2, 2, 2, 2),
    (2, 2, 8, 8, 3, 3, 3, 2, 2, 1, 1),        # stride != padding: the kernels read pad 2, stride 1 with the layer's 4 x 4 output grid
]
# large enough for the tensor-core kernels (batched products with the weight shared by every batch)
TC = [
    (4, 16, 20, 20, 64, 3, 3, 1, 1, 1, 1),    # K = 144, P = 400, Cout = 64
    (3, 32, 12, 16, 72, 3, 3, 1, 1, 1, 1),    # ragged tiles: Cout = 72, P = 192
]


def _data(seed, dt, shape):
    B, C, Hh, W, Co, kh, kw = shape[:7]
    oh, ow, P, K = CC.geometry(*shape)
    rng = np.random.default_rng(seed)
    bound = 1.0 / np.sqrt(K)
    x = H.random_store(rng, dt, B * C * Hh * W, dist="normal")
    w = H.random_store(rng, dt, Co * K, lo=-bound, hi=bound)
    b = H.random_store(rng, dt, Co, lo=-bound, hi=bound)
    g = H.random_store(rng, dt, B * Co * P, dist="normal")
    return x, w, b, g


def _scales(shape):
    B, C, Hh, W, Co, kh, kw = shape[:7]
    oh, ow, P, K = CC.geometry(*shape)
    # magnitude of the sums each result is made of: out ~ sqrt(K) * |w| ~ 1; grad_x ~ sqrt(Co * kh * kw) * |w|; grad_w ~ sqrt(B * P)
    return {"out": 1.0, "grad_x": np.sqrt(Co * kh * kw / K), "grad_w": np.sqrt(B * P), "grad_bias": np.sqrt(B * P)}


def _rel(dt):
    return {"f32": 1e-4, "f64": 1e-10}.get(dt.name, 2e-2)


@pytest.mark.parametrize("dt", [D.F32, D.F64, D.BF16], ids=lambda d: d.name)
@pytest.mark.parametrize("shape", SMALL, ids=lambda s: "x".join(map(str, s)))
def test_oracle_direct_composition_is_a_convolution(oracle, dt, shape):
    from oracle import binding
    x, w, b, g = _data(11, dt, shape)
    binding.set_wide(True)
    try:
        got = CC.compose(oracle, dt, 1, shape, x, w, b, g)
    finally:
        binding.set_wide(False)
    ref = CC.direct_conv_f64(shape, D.decode(x, dt), D.decode(w, dt), D.decode(b, dt), D.decode(g, dt))
    sc = _scales(shape)
    for key in ("out", "grad_x", "grad_w", "grad_bias"):
        r = D.encode(ref[key], dt)
        H.assert_same("conv2d", dt, got[key], r, float_rel=_rel(dt), what=key, scale=sc[key])


def test_reference_call_sequence_differs_from_a_convolution_only_through_its_buffer_labels(oracle):
    """A 1x1 image under a padded 3x3 kernel has one output position (P = 1): the [B][K][P] and [B*P][K] labellings of the column buffer
    coincide, so the literal call sequence (mode 0) must give the convolution too."""
    dt = D.F32
    shape = (5, 4, 1, 1, 3, 3, 3, 1, 1, 1, 1)
    x, w, b, g = _data(12, dt, shape)
    got = CC.compose(oracle, dt, 0, shape, x, w, b, g)
    ref = CC.direct_conv_f64(shape, x, w, b, g)
    H.assert_same("conv2d", dt, got["out"], D.encode(ref["out"], dt), float_rel=1e-5, what="out", scale=1.0)
    # grad_x is not compared: the layer gives col2im num_els = B*C*H*W = 20, so only the first 20 of the 180 column
    # entries are read (crates/maidenx_cpu/src/nn/conv.rs:107,135)
    # the layer labels the [K, Cout] product as [Cout, C, kh, kw]: it is the transpose of the convolution's weight gradient
    gw = D.decode(got["grad_w"], dt).reshape(36, 3).T.reshape(-1)
    assert np.allclose(gw, ref["grad_w"], rtol=1e-5, atol=1e-5)


def _mode_cases():
    ident = lambda s: "x".join(map(str, s))  # noqa: E731
    return [pytest.param(0, s, id="reference-calls-" + ident(s)) for s in LITERAL + TC] + [pytest.param(1, s, id="direct-" + ident(s)) for s in SMALL + TC]


@pytest.mark.gpu
@pytest.mark.parametrize("dt", [D.F32, D.BF16, D.F16, D.F64], ids=lambda d: d.name)
@pytest.mark.parametrize("mode,shape", _mode_cases())
def test_layer_matches_the_oracle_composed_the_same_way(oracle, cuda, dt, mode, shape):
    from oracle import binding
    x, w, b, g = _data(13, dt, shape)
    got = CC.run_layer(dt, mode, shape, x, w, b, g)
    binding.set_wide(True)
    try:
        ref = CC.compose(oracle, dt, mode, shape, x, w, b, g)
    finally:
        binding.set_wide(False)
    H.assert_same("conv2d_im2col", dt, got["cols"], ref["cols"], what="cols")  # a copy: bit-exact
    sc = _scales(shape)
    for key in ("out", "grad_x", "grad_w", "grad_bias"):
        # mode 0 multiplies re-labelled buffers: its sums have the same number of terms, so the same scales serve
        H.assert_same("conv2d", dt, got[key], ref[key], float_rel=_rel(dt), what=f"mode{mode}/{key}", scale=sc[key])


@pytest.mark.gpu
@pytest.mark.parametrize("dt", [D.F32, D.BF16], ids=lambda d: d.name)
@pytest.mark.parametrize("shape", SMALL + TC, ids=lambda s: "x".join(map(str, s)))
def test_direct_layer_is_a_convolution(cuda, dt, shape):
    x, w, b, g = _data(14, dt, shape)
    got = CC.run_layer(dt, 1, shape, x, w, b, g)
    ref = CC.direct_conv_f64(shape, D.decode(x, dt), D.decode(w, dt), D.decode(b, dt), D.decode(g, dt))
    sc = _scales(shape)
    for key in ("out", "grad_x", "grad_w", "grad_bias"):
        H.assert_same("conv2d", dt, got[key], D.encode(ref[key], dt), float_rel=_rel(dt), what=key, scale=sc[key])


@pytest.mark.gpu
def test_literal_call_sequence_is_refused_when_the_swapped_slots_would_mean_a_zero_stride(cuda):
    import ctypes
    from maidenx_b200 import _lib
    lib = _lib.load()
    conv = _lib.MxConv2d(1, 1, 4, 4, 1, 1, 1, 1, 1, 0, 0)
    fwd, _ = _lib.conv2d("f32")
    lib.mx_clear_error()
    fwd(ctypes.byref(conv), 0, 1, 1, None, 1, 1, 1)  # refused before any pointer is touched
    assert lib.mx_last_error() == 3
    lib.mx_clear_error()


@pytest.mark.gpu
@pytest.mark.parametrize("dt", [D.BF16, D.F16], ids=lambda d: d.name)
@pytest.mark.parametrize("shape", [(8, 32, 24, 24, 128, 3, 3, 1, 1, 1, 1), (5, 16, 20, 24, 200, 3, 3, 1, 1, 1, 1)], ids=lambda s: "x".join(map(str, s)))
def test_bias_in_the_product_epilogue_equals_the_separate_add(cuda, dt, shape):
    """Direct form, 16-bit types, shapes the tensor-core kernel takes: the per-channel bias rides in the batched
    product's epilogue (one bias element per output row).  Bit for bit what cuda_matmul followed by cuda_add_inplace
    gives (the op-by-op composition on the same backend), with ragged row tiles (200 channels) as well."""
    x, w, b, g = _data(15, dt, shape)
    got = CC.run_layer(dt, 1, shape, x, w, b, g)
    ref = CC.compose(cuda, dt, 1, shape, x, w, b, g)
    assert np.array_equal(got["out"], ref["out"])
    for key in ("grad_x", "grad_w", "grad_bias"):
        assert np.array_equal(got[key], ref[key]), key


# large enough for the tensor cores, with maps whose rows are no 16-byte multiples (14 x 14, 7 x 7) and regular ones
RAGGED_TC = [
    (5, 24, 14, 14, 136, 3, 3, 1, 1, 1, 1),
    (6, 24, 12, 12, 136, 3, 3, 1, 1, 1, 1),   # P = 144: the weight gradient is one product over batch and positions
    (40, 24, 7, 7, 72, 3, 3, 1, 1, 1, 1),
    (10, 16, 15, 15, 72, 5, 5, 2, 2, 2, 2),
    (40, 128, 7, 7, 72, 3, 3, 1, 1, 1, 1),    # reductions beyond one f16 accumulator run, with the bias in the epilogue
    (40, 129, 8, 8, 72, 3, 3, 1, 1, 1, 1),    # the same with copied weights and tensor stores
    (33, 64, 8, 8, 40, 1, 1, 1, 1, 0, 0),     # many batches of one k-block each, split over CTAs
]


@pytest.mark.gpu
@pytest.mark.parametrize("dt", [D.F32, D.BF16, D.F16], ids=lambda d: d.name)
@pytest.mark.parametrize("shape", RAGGED_TC, ids=lambda s: "x".join(map(str, s)))
def test_direct_layer_on_ragged_maps(cuda, dt, shape):
    """Bounds: f32 1e-5 of the sums' scale (split-tf32 products, f32 sums); 16-bit out and gradients carry at most the
    roundings of the product and of the sum of kh * kw terms."""
    x, w, b, g = _data(15, dt, shape)
    got = CC.run_layer(dt, 1, shape, x, w, b, g)
    ref = CC.direct_conv_f64(shape, D.decode(x, dt), D.decode(w, dt), D.decode(b, dt), D.decode(g, dt))
    sc = _scales(shape)
    for key in ("out", "grad_x", "grad_w", "grad_bias"):
        H.assert_same("conv2d", dt, got[key], D.encode(ref[key], dt), float_rel={"f32": 1e-5}.get(dt.name, 2e-2), what=key, scale=sc[key])


# input channels beyond and below a tile's 128 rows, maps of one and of several row blocks a tile, widths that leave columns of the tile unused, output channels that end inside a k-block,
# kernels that are not square, paddings from none to more than the kernel's half, output maps larger and smaller than the input
IMPLICIT = [
    (3, 64, 14, 14, 72, 3, 3, 1, 1, 1, 1), (2, 130, 9, 31, 64, 3, 3, 1, 1, 1, 1), (5, 8, 7, 7, 8, 5, 5, 1, 1, 2, 2), (2, 200, 28, 28, 136, 3, 3, 1, 1, 1, 1), (1, 64, 17, 130, 136, 1, 3, 1, 1, 0, 1),
    (2, 72, 12, 20, 64, 4, 2, 1, 1, 3, 0), (2, 64, 10, 10, 24, 3, 3, 1, 1, 0, 0), (1, 65, 5, 256, 16, 2, 2, 1, 1, 1, 1), (40, 128, 7, 7, 72, 3, 3, 1, 1, 1, 1), (1, 64, 33, 56, 64, 7, 7, 1, 1, 3, 3),
]


@pytest.mark.gpu
@pytest.mark.parametrize("dt", [D.BF16, D.F16], ids=lambda d: d.name)
@pytest.mark.parametrize("shape", IMPLICIT, ids=lambda s: "x".join(map(str, s)))
def test_input_gradient_without_columns(cuda, dt, shape):
    """One product over taps and channels: next to float64 one rounding of an f32 sum (half a step of the type, and 2^-22 of the sums' scale for the sum itself), and no further off than the columns'
    form, which rounds each of them; nothing else of the layer changes."""
    from maidenx_b200 import _lib
    lib = _lib.load()
    x, w, b, g = _data(16, dt, shape)
    ref = CC.direct_conv_f64(shape, D.decode(x, dt), D.decode(w, dt), D.decode(b, dt), D.decode(g, dt))
    got = {}
    for mode in (0, 2, 1):
        lib.mx_debug_set_conv_implicit(mode)
        try:
            got[mode] = CC.run_layer(dt, 1, shape, x, w, b, g)
        finally:
            lib.mx_debug_set_conv_implicit(1)
    for key in ("out", "grad_w", "grad_bias", "cols"):
        assert np.array_equal(got[0][key], got[2][key]), key
    want = ref["grad_x"].reshape(-1)
    err = {m: np.linalg.norm(D.decode(got[m]["grad_x"], dt) - want) for m in got}
    assert err[2] <= err[0] * 1.0001 and err[1] <= err[0] * 1.0001
    step = 2.0 ** -9 if dt is D.BF16 else 2.0 ** -12
    terms = shape[4] * shape[5] * shape[6]
    assert np.all(np.abs(D.decode(got[2]["grad_x"], dt) - want) <= 1.001 * step * 2 * np.abs(want) + 2.0 ** -20 * _scales(shape)["grad_x"] * np.sqrt(terms) + 1e-7)


@pytest.mark.gpu
@pytest.mark.parametrize("dt", [D.BF16, D.F16], ids=lambda d: d.name)
@pytest.mark.parametrize("what", ["weight_inf", "weight_nan", "many", "gradient", "channel"])
@pytest.mark.parametrize("shape", [(2, 130, 9, 31, 64, 3, 3, 1, 1, 1, 1), (1, 64, 33, 56, 64, 7, 7, 1, 1, 3, 3), (2, 72, 12, 20, 64, 4, 2, 1, 1, 3, 0), (40, 128, 7, 7, 72, 3, 3, 1, 1, 1, 1)],
                         ids=lambda s: "x".join(map(str, s)))
def test_input_gradient_without_columns_keeps_what_is_not_finite(cuda, dt, shape, what):
    """A pixel outside the gradient takes no part in a sum, whatever its weight: infinities and NaNs are where the definition and the columns' form have them, and all else is as without them."""
    from maidenx_b200 import _lib
    lib = _lib.load()
    x, w, b, g = _data(17, dt, shape)
    B, C, Hh, W, Co, kh, kw = shape[:7]
    wf, gf = D.decode(w, dt).astype(np.float64).reshape(Co, C, kh, kw), D.decode(g, dt).astype(np.float64).reshape(B, Co, -1)
    gf[gf == 0.0] = 0.5  # an infinity times one of these would be NaN in either form
    if what == "weight_inf":
        wf[Co - 1, 3, 0, 0], wf[0, C - 1, kh - 1, kw - 1] = np.inf, -np.inf
    elif what == "weight_nan":
        wf[5, 0, kh - 1, 0], wf[Co // 2, C // 2, 0, kw - 1] = np.nan, np.nan
    elif what == "many":
        wf[:, 1], wf[:, 2, 0], wf[3, :, kh // 2, 0] = np.inf, np.nan, -np.inf
    elif what == "gradient":
        gf[0, 1, 0], gf[B - 1, Co - 1, -1], gf[B // 2, 2, 5] = np.inf, np.nan, -np.inf
    else:
        wf[:, 7 % C], gf[0, 3, :4] = np.inf, np.nan
    w, g = D.encode(wf.ravel(), dt), D.encode(gf.ravel(), dt)
    got = {}
    for mode in (0, 2):
        lib.mx_debug_set_conv_implicit(mode)
        try:
            got[mode] = D.decode(CC.run_layer(dt, 1, shape, x, w, b, g)["grad_x"], dt)
        finally:
            lib.mx_debug_set_conv_implicit(1)
    with np.errstate(all="ignore"):
        want = CC.direct_conv_f64(shape, D.decode(x, dt), D.decode(w, dt), D.decode(b, dt), D.decode(g, dt))["grad_x"].reshape(-1)
    for other in (got[0], want):
        assert np.array_equal(np.isnan(got[2]), np.isnan(other)) and np.array_equal(np.isposinf(got[2]), np.isposinf(other)) and np.array_equal(np.isneginf(got[2]), np.isneginf(other))
    fine = np.isfinite(want)
    assert not fine.all() and fine.any()
    step = 2.0 ** -9 if dt is D.BF16 else 2.0 ** -12
    terms = Co * kh * kw
    assert np.all(np.abs(got[2][fine] - want[fine]) <= 1.001 * step * 2 * np.abs(want)[fine] + 2.0 ** -20 * _scales(shape)["grad_x"] * np.sqrt(terms) + 1e-7)


@pytest.mark.gpu
@pytest.mark.parametrize("dt", [D.BF16, D.F16], ids=lambda d: d.name)
def test_literal_call_sequence_is_these_calls(cuda, dt):
    """Mode 0 gives what the reference's calls give one after the other, bit for bit: here a sum in another order would not (each row holds a large number and its negative)."""
    shape = (4, 3, 100, 223, 16, 3, 3, 1, 1, 1, 1)
    x, w, b, _ = _data(18, dt, shape)
    rng = np.random.default_rng(18)
    g = rng.standard_normal((4 * 16 * 100, 223)) * 1e-3
    at = np.argsort(rng.random(g.shape), axis=1)[:, :2]
    np.put_along_axis(g, at, np.array([30000.0, -30000.0]), axis=1)
    g = D.encode(g.ravel(), dt)
    got, want = CC.run_layer(dt, 0, shape, x, w, b, g), CC.compose(cuda, dt, 0, shape, x, w, b, g)
    assert np.array_equal(got["grad_bias"], want["grad_bias"])


# batch, channels, height, width: lanes a row by vectors (4, 8, 16, 32) and by elements (8, 16, 32), one and two trips, many planes of middle sizes - and, from "sums" on, maps whose two sums stay as they are
BIAS_SUMS = [(1, 16, 13, 8), (3, 40, 33, 32), (2, 8, 31, 56), (1, 9, 15, 104), (1, 5, 7, 136), (2, 3, 4, 480), (7, 40, 16, 7), (5, 64, 14, 14), (1, 33, 4, 63), (32, 64, 20, 48), (32, 64, 44, 48), (64, 32, 33, 33), (64, 32, 33, 41),
             "sums", (1, 16, 112, 112), (1, 16, 55, 55), (1, 64, 56, 56), (2, 3, 300, 200), (100, 90, 7, 7), (64, 32, 28, 28), (64, 32, 9, 64)]


@pytest.mark.gpu
@pytest.mark.parametrize("dt", [D.BF16, D.F16], ids=lambda d: d.name)
@pytest.mark.parametrize("case", [c for c in BIAS_SUMS if c != "sums"], ids=str)
def test_bias_gradient_s_sums(cuda, dt, case):
    """Whole numbers, whose sums are exact in f32: the bits of the sums one after the other, whichever way they are taken.  Where a warp a plane does not pay they are those calls, and then also
    have their bits for rows that a sum in another order would change."""
    B, Co, h, w = case
    shape = (B, 1, h, w, Co, 1, 1, 1, 1, 0, 0)
    rng = np.random.default_rng(19)
    data = [rng.integers(-8, 9, (B * Co * h, w)).astype(np.float64)]
    if BIAS_SUMS.index(case) > BIAS_SUMS.index("sums"):
        g = rng.standard_normal(data[0].shape) * 1e-3
        np.put_along_axis(g, np.argsort(rng.random(g.shape), axis=1)[:, :2], np.array([30000.0, -30000.0]), axis=1)
        data.append(g)
    x, wt = D.encode(rng.standard_normal(B * h * w), dt), D.encode(rng.standard_normal(Co), dt)
    for g in data:
        g = D.encode(g.ravel(), dt)
        got, want = CC.run_layer(dt, 1, shape, x, wt, None, g), CC.compose(cuda, dt, 1, shape, x, wt, None, g)
        assert np.array_equal(got["grad_bias"], want["grad_bias"])


# A wide kernel on planes of whole lines, with pixels of grad_out that are not in whole 32 bytes and that are;
# a few output channels on planes of whole lines, a ragged plane with many, more rows of weights than columns pay for - and maps, ragged or large, whose columns cost more
ROUTES = [((4, 80, 64, 64, 248, 5, 5, 1, 1, 2, 2), "columns"), ((3, 184, 56, 56, 160, 5, 5, 1, 1, 2, 2), "one product"),
          ((11, 88, 56, 56, 8, 3, 3, 1, 1, 1, 1), "columns"), ((14, 152, 28, 28, 408, 3, 3, 1, 1, 0, 0), "columns"), ((13, 80, 28, 28, 288, 3, 3, 1, 1, 1, 1), "columns"),
          ((36, 224, 14, 14, 112, 3, 3, 1, 1, 1, 1), "one product"), ((8, 192, 56, 56, 64, 3, 3, 1, 1, 1, 1), "one product"), ((42, 153, 14, 14, 16, 7, 7, 1, 1, 0, 0), "one product")]


@pytest.mark.gpu
@pytest.mark.parametrize("shape,way", ROUTES, ids=str)
def test_which_input_gradients_go_without_columns(cuda, shape, way):
    """The rule on sizes takes the way that was measured to be the faster one: the bits of the switch for that way, which differ where sums are rounded once and not once a tap."""
    from maidenx_b200 import _lib
    lib, dt = _lib.load(), D.BF16
    rng = np.random.default_rng(20)
    oh, ow, P, K = CC.geometry(*shape)
    B, C, Hh, W, Co = shape[:5]
    x, w, g = (D.encode(rng.standard_normal(n).astype(np.float32), dt) for n in (B * C * Hh * W, Co * K, B * Co * P))
    got = {}
    for mode in (0, 1, 2):
        lib.mx_debug_set_conv_implicit(mode)
        try:
            got[mode] = CC.run_layer(dt, 1, shape, x, w, None, g)["grad_x"]
        finally:
            lib.mx_debug_set_conv_implicit(1)
    assert not np.array_equal(got[0], got[2]) and np.array_equal(got[1], got[0 if way == "columns" else 2])
