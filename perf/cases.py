"""The work that users of this op layer have it do, as timed and checked cases.

Every case is one pass through the entry points a program calls: `device.dispatch` (metadata block uploaded, op called,
block freed, as maidenx_core does around each op), the Conv2d layer of `mx_conv2d_*`, and the MLP engine.  Sizes are
those of the README example, the benchmark's configurations and generic ones of the same families, regular and ragged:

  readme       the README example's training step: 17 small f32 ops, where launches and dispatch are the time
  mlp          the MLP engine's training step (forward, MSE, backward, SGD), small and at the benchmark's size
  linear       one Linear layer op by op: x . W^T + b, and the three gradients autograd issues
  bmm          a batched product and its backward (attention scores, per-head projections)
  conv         Conv2d forward and backward: the benchmark's 56 x 56 layer and the 14 x 14 maps deeper in such a network
  layer_norm   the normalisation composed from reductions along the rows and broadcasts
  softmax      scaled softmax over a dim of a 3-d tensor and its backward
  affine       per-channel scale and shift of image batches and their gradients
  matrix       the single-op sweeps' layouts on one matrix: flat, transposed and broadcast operands, both reductions
"""
import ctypes
import math

import torch

from maidenx_b200 import _lib, device
from maidenx_b200.mlp import Mlp

TORCH = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
SIZE = {"f32": 4, "bf16": 2, "f16": 2}
LR = 1e-3


def listed():
    return [
        # the smallest work: the reference's own training example at its own size
        {"name": "readme_step", "kind": "readme", "dtype": "f32", "rows": 10000, "features": 3},
        # a small network on the training engine: launch-bound products and passes
        {"name": "mlp_small", "kind": "mlp", "dtype": "bf16", "layers": 2, "dim": 1024, "batch": 512},
        # the benchmark's headline step
        {"name": "mlp_large", "kind": "mlp", "dtype": "bf16", "layers": 4, "dim": 8192, "batch": 16384},
        # a hidden layer of a digit classifier
        {"name": "linear_f32_small", "kind": "linear", "dtype": "f32", "batch": 128, "fan_in": 784, "fan_out": 300},
        # a wide layer whose sizes are multiples of nothing: a last, incomplete batch and a vocabulary-like output
        {"name": "linear_bf16_ragged", "kind": "linear", "dtype": "bf16", "batch": 4099, "fan_in": 1000, "fan_out": 1543},
        # attention scores of a batch of 16 x 8 heads
        {"name": "bmm_bf16", "kind": "bmm", "dtype": "bf16", "batch": 128, "m": 384, "n": 384, "k": 64},
        # the benchmark's Conv2d layer
        {"name": "conv_bf16_56", "kind": "conv", "dtype": "bf16", "n": 64, "c": 256, "hw": 56, "co": 256, "k": 3, "stride": 1, "pad": 1},
        # the same network two stages deeper
        {"name": "conv_f32_14", "kind": "conv", "dtype": "f32", "n": 32, "c": 128, "hw": 14, "co": 256, "k": 3, "stride": 1, "pad": 1},
        # normalisation of a batch of odd-length rows
        {"name": "layer_norm_f32", "kind": "layer_norm", "dtype": "f32", "rows": 8191, "cols": 1023},
        # attention probabilities over 197 positions (a 14 x 14 grid and one more)
        {"name": "softmax_bf16", "kind": "softmax", "dtype": "bf16", "batch": 192, "rows": 197, "cols": 197, "dim": 2},
        # scale and shift of the last feature maps of an image network (7 x 7)
        {"name": "affine_bf16_7", "kind": "affine", "dtype": "bf16", "n": 256, "c": 512, "hw": 7},
        # the sweeps' layouts at a size of the sweeps
        {"name": "matrix_f32", "kind": "matrix", "dtype": "f32", "rows": 8192, "cols": 16384},
    ]


def _log(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]; half of them rounded to a multiple of 8."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.5 and v >= 8:
        v -= v % 8
    return min(hi, max(lo, v))


def draw(rng):
    kind = rng.choice(["readme", "mlp", "linear", "bmm", "conv", "layer_norm", "softmax", "affine", "matrix"])
    dtype = rng.choice(["f32", "bf16", "f16"])
    while True:
        if kind == "readme":
            c = {"kind": kind, "dtype": "f32", "rows": _log(rng, 1000, 20000), "features": rng.randint(1, 16)}
        elif kind == "mlp":
            c = {"kind": kind, "dtype": "bf16", "layers": rng.randint(1, 4), "dim": 8 * _log(rng, 16, 512), "batch": _log(rng, 32, 16384)}
        elif kind == "linear":
            c = {"kind": kind, "dtype": dtype, "batch": _log(rng, 32, 16384), "fan_in": _log(rng, 8, 4096), "fan_out": _log(rng, 8, 4096)}
        elif kind == "bmm":
            c = {"kind": kind, "dtype": dtype, "batch": _log(rng, 2, 256), "m": _log(rng, 16, 1024), "n": _log(rng, 16, 1024), "k": _log(rng, 16, 256)}
        elif kind == "conv":
            k = rng.choice([1, 3, 3, 5, 7])
            c = {"kind": kind, "dtype": dtype, "n": rng.randint(1, 64), "c": _log(rng, 3, 256), "hw": rng.choice([7, 14, 28, 56, 112, rng.randint(7, 112)]),
                 "co": _log(rng, 16, 512), "k": k, "stride": rng.choice([1, 1, 2]), "pad": k // 2}
        elif kind == "layer_norm":
            c = {"kind": kind, "dtype": dtype, "rows": _log(rng, 64, 32768), "cols": _log(rng, 64, 8192)}
        elif kind == "softmax":
            c = {"kind": kind, "dtype": dtype, "batch": _log(rng, 1, 256), "rows": _log(rng, 16, 1024), "cols": _log(rng, 16, 1024), "dim": rng.choice([2, 2, 1])}
        elif kind == "affine":
            c = {"kind": kind, "dtype": dtype, "n": _log(rng, 1, 256), "c": _log(rng, 8, 512), "hw": rng.choice([7, 14, 28, 56, 112, rng.randint(7, 112)])}
        else:
            c = {"kind": kind, "dtype": dtype, "rows": _log(rng, 512, 16384), "cols": _log(rng, 512, 16384)}
        w = work(c)
        # a product on the CUDA cores runs three orders slower than one on the tensor cores: bound what a drawn case may cost either way
        if w["bytes"] <= 6e9 and w["flops"] <= (2.4e13 if kind == "mlp" else 1.2e12) and _conv_cols(c) <= 4e8:
            return c


def _conv_out(c):
    return (c["hw"] + 2 * c["pad"] - c["k"]) // c["stride"] + 1


def _conv_cols(c):
    return c["n"] * c["c"] * c["k"] ** 2 * _conv_out(c) ** 2 if c["kind"] == "conv" else 0


# ---- op calls ------------------------------------------------------------------------------------------------------
def _strides(dims):
    st, acc = [], 1
    for d in reversed(dims):
        st.append(acc)
        acc *= d
    return st[::-1]


def _p(t):
    return t.data_ptr()


def _const(dtype, v):
    """A by-value scalar: 16-bit floats travel as their bit pattern."""
    return v if dtype == "f32" else int(torch.tensor(v, dtype=TORCH[dtype]).view(torch.int16)) & 0xFFFF


def _binary(op, dt, dims, sa, sb, a, b, out):
    device.dispatch(op, dt, [*dims, *sa, *sb, 0, 0], math.prod(dims), len(dims), "META", _p(a), _p(b), _p(out))
    return out


def _unary(op, dt, dims, st, x, out, *const):
    device.dispatch(op, dt, [*dims, *st, 0], math.prod(dims), len(dims), "META", _p(x), *const, _p(out))
    return out


def _reduce(op, dt, dims, dim, x, out):
    st = _strides(dims)
    device.dispatch(op, dt, [*dims, *st, dims[dim], st[dim], 0], math.prod(dims), len(dims), 1, "META", _p(x), _p(out))
    return out


def _fold(dt, dims, out_dims, x, out):
    device.dispatch("sum_to_shape", dt, [*dims, *_strides(dims), *out_dims, 0], math.prod(dims), len(dims), "META", _p(x), _p(out))
    return out


def _matmul(dt, od, ad, bd, sa, sb, a, b, out):
    device.dispatch("matmul", dt, [len(od), len(ad), len(bd), *od, *ad, *bd, *sa, *sb, 0, 0], math.prod(od), "META", _p(a), _p(b), _p(out))
    return out


class _EngineArray:
    """Device memory of an MLP engine as an array that torch can wrap; a tensor made of it keeps the engine alive."""

    def __init__(self, engine, ptr, count, typestr):
        self.engine = engine
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (count,), "typestr": typestr, "version": 3}


def _engine(m, ptr, count, typestr="<f4"):
    """f32, or bf16 for the two-byte type."""
    t = torch.as_tensor(_EngineArray(m, ptr, count, typestr), device="cuda")
    return t.view(torch.bfloat16) if typestr == "<i2" else t


# ---- inputs --------------------------------------------------------------------------------------------------------
def _inputs(case, seed):
    """The tensors of a case, from the seed alone: activations and gradients are normal, weights scaled by their fan-in."""
    g = torch.Generator(device="cuda").manual_seed(seed * 7919 + 13)
    dt = TORCH[case["dtype"]]

    def normal(*shape, scale=1.0):
        return (torch.randn(shape, device="cuda", generator=g) * scale).to(dt)

    k = case["kind"]
    if k == "readme":
        n, f = case["rows"], case["features"]
        x = torch.rand((n, f), device="cuda", generator=g)
        y = x.sum(1, keepdim=True) * 0.1 + 0.01 * torch.randn((n, 1), device="cuda", generator=g)
        return {"x": x, "y": y, "w": normal(1, f, scale=0.3), "b": normal(1, scale=0.1), "one": torch.ones(1, device="cuda")}
    if k == "mlp":
        b, d = case["batch"], case["dim"]
        t = {"x": normal(b, d), "y": normal(b, d)}
        t["w"] = [(torch.rand((d, d), device="cuda", generator=g) * 2 - 1) / d ** 0.5 for _ in range(case["layers"])]
        t["b"] = [(torch.rand(1, device="cuda", generator=g) * 2 - 1) / d ** 0.5 for _ in range(case["layers"])]
        return t
    if k == "linear":
        b, i, o = case["batch"], case["fan_in"], case["fan_out"]
        return {"x": normal(b, i), "w": normal(o, i, scale=i ** -0.5), "b": normal(o), "g": normal(b, o)}
    if k == "bmm":
        b, m, n, kk = case["batch"], case["m"], case["n"], case["k"]
        return {"a": normal(b, m, kk), "b": normal(b, kk, n), "g": normal(b, m, n)}
    if k == "conv":
        n, c, hw, co, kk, o = case["n"], case["c"], case["hw"], case["co"], case["k"], _conv_out(case)
        return {"x": normal(n, c, hw, hw), "w": normal(co, c, kk, kk, scale=(c * kk * kk) ** -0.5), "b": normal(co), "g": normal(n, co, o, o)}
    if k == "layer_norm":
        r, c = case["rows"], case["cols"]
        return {"x": normal(r, c) + 0.5, "gamma": normal(c, scale=0.1) + 1, "beta": normal(c, scale=0.1)}
    if k == "softmax":
        b, r, c = case["batch"], case["rows"], case["cols"]
        return {"x": normal(b, r, c, scale=8.0), "g": normal(b, r, c)}
    if k == "affine":
        n, c, hw = case["n"], case["c"], case["hw"]
        return {"x": normal(n, c, hw, hw), "scale": normal(c, scale=0.2) + 1, "shift": normal(c, scale=0.2), "g": normal(n, c, hw, hw)}
    r, c = case["rows"], case["cols"]
    return {"a": normal(r, c), "b": normal(r, c), "t": normal(c, r), "row": normal(c)}


def prepare(case, seed):
    t = _inputs(case, seed)
    dt = TORCH[case["dtype"]]

    def new(*shape):
        return torch.empty(shape, device="cuda", dtype=dt)

    k = case["kind"]
    s = {"case": case, "in": t}
    if k == "readme":
        n, f = case["rows"], case["features"]
        s["buf"] = [new(n) for _ in range(9)] + [new(1) for _ in range(6)] + [new(f) for _ in range(3)]
    elif k == "mlp":
        m = Mlp(case["layers"], case["dim"], case["batch"], case["dtype"], seed=1)
        d = case["dim"]
        grads = [(_engine(m, m.ptr("weight_grad", l), d * d, "<i2"), _engine(m, m.ptr("bias_grad", l), 1, "<i2")) for l in range(case["layers"])]
        for l in range(case["layers"]):
            grads[l][0].zero_()
            grads[l][1].zero_()
            _engine(m, m.ptr("master_weight", l), d * d).copy_(t["w"][l].flatten())
            _engine(m, m.ptr("master_bias", l), 1).copy_(t["b"][l])
            m.sgd_layer(l, 0.0)  # the engine's 16-bit copies follow its master weights
        t.pop("w")
        s.update(mlp=m, grads=grads, pred=_engine(m, m.ptr("output"), case["batch"] * d, "<i2"), loss=_engine(m, m.ptr("loss_ptr"), 1))
    elif k == "linear":
        b, i, o = case["batch"], case["fan_in"], case["fan_out"]
        s.update(z=new(b, o), y=new(b, o), dx=new(b, i), dw=new(o, i), db=new(1, o))
    elif k == "bmm":
        b, m, n, kk = case["batch"], case["m"], case["n"], case["k"]
        s.update(c=new(b, m, n), da=new(b, m, kk), db=new(b, kk, n))
    elif k == "conv":
        conv = _lib.MxConv2d(case["n"], case["c"], case["hw"], case["hw"], case["co"], case["k"], case["k"], case["stride"], case["stride"], case["pad"], case["pad"])
        fwd, bwd = _lib.conv2d(case["dtype"])
        lib, ref = _lib.load(), ctypes.byref(conv)
        ws = max(lib.mx_conv2d_workspace_elems(ref, 1, 0), lib.mx_conv2d_workspace_elems(ref, 1, 1))
        s.update(conv=conv, fwd=fwd, bwd=bwd, cols=new(lib.mx_conv2d_cols_elems(ref)), ws=new(ws), y=torch.empty_like(t["g"]), dx=torch.empty_like(t["x"]),
                 dw=torch.empty_like(t["w"]), db=torch.empty_like(t["b"]))
    elif k == "layer_norm":
        r, c = case["rows"], case["cols"]
        s.update(buf=[new(r, c) for _ in range(3)], col=[new(r) for _ in range(4)], y=new(r, c))
    elif k == "softmax":
        b, r, c = case["batch"], case["rows"], case["cols"]
        s.update(buf=[new(b, r, c) for _ in range(2)], red=new(b * (r if case["dim"] == 2 else c)), p=new(b, r, c), dx=new(b, r, c))
    elif k == "affine":
        s.update(buf=[torch.empty_like(t["x"]) for _ in range(2)], y=torch.empty_like(t["x"]), dx=torch.empty_like(t["x"]), dscale=new(case["c"]), dshift=new(case["c"]))
    else:
        r, c = case["rows"], case["cols"]
        s.update(out=[new(r, c) for _ in range(4)], col=[new(c) for _ in range(2)], row=[new(r) for _ in range(2)])
    return s


# ---- passes --------------------------------------------------------------------------------------------------------
def run(state):
    return globals()["_run_" + state["case"]["kind"]](state)


def _run_readme(s):
    n, f, t, b = s["case"]["rows"], s["case"]["features"], s["in"], s["buf"]
    col = [n, 1, 1, 1]
    z, pred, diff, sq, s1, p1, two, dpred = b[:8]
    total, loss, g, db, sb, nb = b[9:15]
    dw, sw, nw = b[15:18]
    _matmul("f32", [n, 1], [n, f], [f, 1], [f, 1], [1, f], t["x"], t["w"], z)
    _binary("add", "f32", [n, 1], [1, 1], [0, 0], z, t["b"], pred)
    _binary("sub", "f32", [n, 1], [1, 1], [1, 1], pred, t["y"], diff)
    _unary("pow", "f32", [n, 1], [1, 1], diff, sq, 2.0)
    _reduce("sum", "f32", [n, 1], 1, sq, s1)
    _reduce("sum", "f32", [n], 0, s1, total)
    _unary("div_scalar", "f32", [1], [1], total, loss, float(n))
    _unary("div_scalar", "f32", [1], [1], t["one"], g, float(n))
    _unary("pow", "f32", [n, 1], [1, 1], diff, p1, 1.0)
    _unary("mul_scalar", "f32", [n, 1], [1, 1], p1, two, 2.0)
    _binary("mul", "f32", [n, 1], [1, 1], [0, 0], two, g, dpred)
    _fold("f32", [n, 1], [1, 1], dpred, db)
    _matmul("f32", [1, f], [1, n], [n, f], [1, 1], [f, 1], dpred, t["x"], dw)
    _unary("mul_scalar", "f32", [f], [1], dw, sw, 0.01)
    _binary("sub", "f32", [f], [1], [1], t["w"], sw, nw)
    _unary("mul_scalar", "f32", [1], [1], db, sb, 0.01)
    _binary("sub", "f32", [1], [1], [1], t["b"], sb, nb)
    return {"loss": loss, "dw": dw, "db": db, "w": nw, "b": nb}


def _run_mlp(s):
    s["mlp"].train_step(_p(s["in"]["x"]), _p(s["in"]["y"]), LR)
    return {"pred": s["pred"], "loss": s["loss"], "dw": [g[0] for g in s["grads"]], "db": [g[1] for g in s["grads"]]}


def _run_linear(s):
    c, t = s["case"], s["in"]
    dt, b, i, o = c["dtype"], c["batch"], c["fan_in"], c["fan_out"]
    _matmul(dt, [b, o], [b, i], [i, o], [i, 1], [1, i], t["x"], t["w"], s["z"])  # the transposed view of W
    _binary("add", dt, [b, o], [o, 1], [0, 1], s["z"], t["b"], s["y"])
    _matmul(dt, [b, i], [b, o], [o, i], [o, 1], [i, 1], t["g"], t["w"], s["dx"])
    _matmul(dt, [o, i], [o, b], [b, i], [1, o], [i, 1], t["g"], t["x"], s["dw"])  # the transposed view of g
    _fold(dt, [b, o], [1, o], t["g"], s["db"])
    return {"y": s["y"], "dx": s["dx"], "dw": s["dw"], "db": s["db"]}


def _run_bmm(s):
    c, t = s["case"], s["in"]
    b, m, n, k = c["batch"], c["m"], c["n"], c["k"]
    od, ad, bd = [b, m, n], [b, m, k], [b, k, n]
    _matmul(c["dtype"], od, ad, bd, _strides(ad), _strides(bd), t["a"], t["b"], s["c"])
    meta = [3, 3, 3, *od, *ad, *bd, *_strides(ad), *_strides(bd), 0, 0]
    device.dispatch("matmul_backward", c["dtype"], meta, b * m * k, b * k * n, "META", _p(t["g"]), _p(t["a"]), _p(t["b"]), _p(s["da"]), _p(s["db"]))
    return {"c": s["c"], "da": s["da"], "db": s["db"]}


def _run_conv(s):
    t, conv = s["in"], ctypes.byref(s["conv"])
    s["fwd"](conv, 1, _p(t["x"]), _p(t["w"]), _p(t["b"]), _p(s["cols"]), _p(s["ws"]), _p(s["y"]))
    s["bwd"](conv, 1, _p(t["g"]), _p(t["w"]), _p(s["cols"]), _p(s["ws"]), _p(s["dx"]), _p(s["dw"]), _p(s["db"]))
    if device.last_error():
        raise device.CudaError(device.last_error())
    return {"y": s["y"], "dx": s["dx"], "dw": s["dw"], "db": s["db"]}


def _run_layer_norm(s):
    c, t = s["case"], s["in"]
    dt, d = c["dtype"], [c["rows"], c["cols"]]
    st, per_row, per_col = [d[1], 1], [1, 0], [0, 1]
    diff, sq, xhat = s["buf"]
    mean, var, vare, std = s["col"]
    _reduce("mean", dt, d, 1, t["x"], mean)
    _binary("sub", dt, d, st, per_row, t["x"], mean, diff)
    _unary("square", dt, d, st, diff, sq)
    _reduce("mean", dt, d, 1, sq, var)
    _unary("add_scalar", dt, [d[0]], [1], var, vare, _const(dt, 1e-5))
    _unary("sqrt", dt, [d[0]], [1], vare, std)
    _binary("div", dt, d, st, per_row, diff, std, xhat)
    _binary("mul", dt, d, st, per_col, xhat, t["gamma"], sq)
    _binary("add", dt, d, st, per_col, sq, t["beta"], s["y"])
    return {"y": s["y"], "mean": mean, "var": var}


def _run_softmax(s):
    c, t = s["case"], s["in"]
    dt, d, dim = c["dtype"], [c["batch"], c["rows"], c["cols"]], c["dim"]
    st = _strides(d)
    scaled, gp = s["buf"]
    per = [d[1], 1, 0] if dim == 2 else [d[2], 0, 1]
    _unary("mul_scalar", dt, d, st, t["x"], scaled, _const(dt, 0.125))
    device.dispatch("softmax", dt, [*d, *st, 0], math.prod(d), 3, dim, "META", _p(scaled), _p(s["p"]))
    _binary("mul", dt, d, st, st, t["g"], s["p"], gp)
    _reduce("sum", dt, d, dim, gp, s["red"])
    _binary("sub", dt, d, st, per, t["g"], s["red"], gp)
    _binary("mul", dt, d, st, st, gp, s["p"], s["dx"])
    return {"p": s["p"], "dx": s["dx"]}


def _run_affine(s):
    c, t = s["case"], s["in"]
    dt, d = c["dtype"], [c["n"], c["c"], c["hw"], c["hw"]]
    st, per = _strides(d), [0, 1, 0, 0]
    u, v = s["buf"]
    _binary("mul", dt, d, st, per, t["x"], t["scale"], u)
    _binary("add", dt, d, st, per, u, t["shift"], v)
    _unary("relu", dt, d, st, v, s["y"])
    _binary("mul", dt, d, st, per, t["g"], t["scale"], s["dx"])
    _binary("mul", dt, d, st, st, t["g"], t["x"], u)
    _fold(dt, d, [1, d[1], 1, 1], u, s["dscale"])
    _fold(dt, d, [1, d[1], 1, 1], t["g"], s["dshift"])
    return {"y": s["y"], "dx": s["dx"], "dscale": s["dscale"], "dshift": s["dshift"]}


def _run_matrix(s):
    c, t = s["case"], s["in"]
    dt, d = c["dtype"], [c["rows"], c["cols"]]
    st = [d[1], 1]
    _binary("add", dt, d, st, st, t["a"], t["b"], s["out"][0])
    _binary("mul", dt, d, [1, d[0]], st, t["t"], t["b"], s["out"][1])  # the transposed view of t
    _binary("div", dt, d, st, [0, 1], t["a"], t["row"], s["out"][2])
    _unary("gelu", dt, d, st, t["a"], s["out"][3])
    _reduce("sum", dt, d, 0, t["a"], s["col"][0])
    _reduce("max", dt, d, 0, t["b"], s["col"][1])
    _reduce("mean", dt, d, 1, t["a"], s["row"][0])
    _reduce("sum", dt, d, 1, t["b"], s["row"][1])
    return {"out": s["out"], "col": s["col"], "row": s["row"]}


# ---- what a pass cannot do without ---------------------------------------------------------------------------------
def work(case):
    """Each input read once, each output written once, and the products' operations."""
    k, e = case["kind"], SIZE[case["dtype"]]
    if k == "readme":
        n, f = case["rows"], case["features"]
        return {"bytes": 4 * (n * f + n + 3 * f + 5), "flops": 4 * n * f + 8 * n}
    if k == "mlp":
        b, d, l = case["batch"], case["dim"], case["layers"]
        # master weights read and written, 16-bit weights read and written, gradients and activations written
        return {"bytes": l * d * d * (4 + 4 + 2 + 2 + 2) + 2 * b * d * (3 + l), "flops": 2 * b * d * d * (3 * l - 1)}
    if k == "linear":
        b, i, o = case["batch"], case["fan_in"], case["fan_out"]
        return {"bytes": e * (2 * b * i + 2 * o * i + 2 * o + 2 * b * o), "flops": 6 * b * i * o}
    if k == "bmm":
        b, m, n, kk = case["batch"], case["m"], case["n"], case["k"]
        return {"bytes": 2 * e * b * (m * kk + kk * n + m * n), "flops": 6 * b * m * n * kk}
    if k == "conv":
        n, c, hw, co, kk, o = case["n"], case["c"], case["hw"], case["co"], case["k"], _conv_out(case)
        return {"bytes": 2 * e * (n * c * hw * hw + co * c * kk * kk + co + n * co * o * o), "flops": 6 * n * o * o * co * c * kk * kk}
    if k == "layer_norm":
        r, c = case["rows"], case["cols"]
        return {"bytes": e * (2 * r * c + 2 * c + 2 * r), "flops": 8 * r * c}
    if k == "softmax":
        n = case["batch"] * case["rows"] * case["cols"]
        return {"bytes": 4 * e * n, "flops": 8 * n}
    if k == "affine":
        n = case["n"] * case["c"] * case["hw"] ** 2
        return {"bytes": e * (4 * n + 4 * case["c"]), "flops": 7 * n}
    n = case["rows"] * case["cols"]
    return {"bytes": e * (7 * n + 3 * case["cols"] + 2 * case["rows"]), "flops": 12 * n}


def tolerance(case):
    return {"rel": 2e-5 if case["dtype"] == "f32" else 1e-2}


# ---- the same in 64 bits -------------------------------------------------------------------------------------------
def exact(case, seed):
    t = {n: [x.double() for x in v] if isinstance(v, list) else v.double() for n, v in _inputs(case, seed).items()}
    k = case["kind"]
    if k == "readme":
        n = case["rows"]
        diff = t["x"] @ t["w"].T + t["b"] - t["y"]
        d = 2 * diff / n
        dw, db = (d.T @ t["x"]).flatten(), d.sum().reshape(1)
        return {"loss": (diff ** 2).sum().reshape(1) / n, "dw": dw, "db": db, "w": t["w"].flatten() - 0.01 * dw, "b": t["b"] - 0.01 * db}
    if k == "mlp":
        layers = case["layers"]
        w = [x.bfloat16().double() for x in t["w"]]
        b = [x.bfloat16().double() for x in t["b"]]
        acts, pre = [t["x"]], []
        for l in range(layers):
            u = acts[-1] @ w[l].T + b[l]
            pre.append(u)
            acts.append(torch.nn.functional.gelu(u, approximate="tanh"))
        pred = pre[-1]
        diff = pred - t["y"]
        du = 2 * diff / diff.numel()
        dw, db = [None] * layers, [None] * layers
        for l in reversed(range(layers)):
            dw[l], db[l] = (du.T @ acts[l]).flatten(), du.sum().reshape(1)
            if l:
                u = pre[l - 1]
                th = torch.tanh(0.7978845608028654 * (u + 0.044715 * u ** 3))
                du = (du @ w[l]) * (0.5 * (1 + th) + 0.5 * u * (1 - th * th) * 0.7978845608028654 * (1 + 3 * 0.044715 * u * u))
        return {"pred": pred.flatten(), "loss": (diff ** 2).mean().reshape(1), "dw": dw, "db": db}
    if k == "linear":
        return {"y": t["x"] @ t["w"].T + t["b"], "dx": t["g"] @ t["w"], "dw": t["g"].T @ t["x"], "db": t["g"].sum(0, keepdim=True)}
    if k == "bmm":
        return {"c": t["a"] @ t["b"], "da": t["g"] @ t["b"].transpose(1, 2), "db": t["a"].transpose(1, 2) @ t["g"]}
    if k == "conv":
        n, kk, st, pad, o = case["n"], case["k"], case["stride"], case["pad"], _conv_out(case)
        w = t["w"].flatten(1)
        y, dx, dw = torch.empty_like(t["g"]), torch.empty_like(t["x"]), torch.zeros_like(w)
        for i in range(0, n, 8):  # unfold, product and fold, a few images at a time
            x, g = t["x"][i:i + 8], t["g"][i:i + 8].flatten(2)
            cols = torch.nn.functional.unfold(x, kk, padding=pad, stride=st)
            y[i:i + 8] = (w @ cols).view(-1, case["co"], o, o) + t["b"].view(1, -1, 1, 1)
            dw += (g @ cols.transpose(1, 2)).sum(0)
            dx[i:i + 8] = torch.nn.functional.fold(w.T @ g, (case["hw"], case["hw"]), kk, padding=pad, stride=st)
        return {"y": y, "dx": dx, "dw": dw.view_as(t["w"]), "db": t["g"].sum((0, 2, 3))}
    if k == "layer_norm":
        mean = t["x"].mean(1, keepdim=True)
        var = ((t["x"] - mean) ** 2).mean(1, keepdim=True)
        return {"y": (t["x"] - mean) / (var + 1e-5).sqrt() * t["gamma"] + t["beta"], "mean": mean.flatten(), "var": var.flatten()}
    if k == "softmax":
        p = torch.softmax(t["x"] * 0.125, case["dim"])
        return {"p": p, "dx": p * (t["g"] - (t["g"] * p).sum(case["dim"], keepdim=True))}
    if k == "affine":
        per = (1, -1, 1, 1)
        return {"y": torch.relu(t["x"] * t["scale"].view(per) + t["shift"].view(per)), "dx": t["g"] * t["scale"].view(per), "dscale": (t["g"] * t["x"]).sum((0, 2, 3)),
                "dshift": t["g"].sum((0, 2, 3))}
    a, b = t["a"], t["b"]
    return {"out": [a + b, t["t"].T * b, a / t["row"], torch.nn.functional.gelu(a, approximate="tanh")], "col": [a.sum(0), b.amax(0)], "row": [a.mean(1), b.sum(1)]}
