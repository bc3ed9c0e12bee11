"""What the library is timed on: the calls a user's program makes, from one small inference call to a whole
training step, each through the public entry points.

Five kinds of case:

``linear``   ``ops.linear_*``   forward, or forward + weight and bias gradient + input gradient
``conv``     ``ops.conv_*``     the same for Conv2d / ConvTranspose2d; fp16 NHWC (how the nets of ``train.py`` keep
                                their activations) or fp32 NCHW (the reference's tensors, 3xTF32 arithmetic)
``dropin``   ``_nectarml.*``    the reference's own host ops: device pointers in, a pointer out; convolutions as its
``matmul``                      autograd calls them (with ``half_precision`` the forward runs on fp16 operands, the
                                backward stays fp32), and its batched matmul
``block``    ``train.*``        a bottleneck residual block: forward, backward, finiteness check, SGD-momentum update
``step``     ``train.*``        one optimisation step of a net; issued call by call or replayed from a CUDA graph

Layer sizes are those of the benchmark's sweeps and of the two nets, or generic ones around them.  The ResNet-50 step
is here as its stem and its blocks: through all 53 normalised layers at random weights one fp16 value that rounds the
other way changes the gradients by tens of percents, so the results of two correct programs could not be compared.
"""
import math

import torch

from nectarml_b200 import _nectarml, ops, train
from nectarml_b200.ops import ConvGeometry

DEV = "cuda"


def _linear(name, rows, fin, fout, dtype, passes):
    return {"name": name, "kind": "linear", "rows": rows, "fin": fin, "fout": fout, "dtype": dtype, "passes": passes}


def _conv(name, kind, dtype, batch, c_in, hw, c_out, k, stride, pad, transposed=False, bias=True, passes="train"):
    """``passes``: fwd; fwd+dw (a first layer: nobody wants the gradient of the image); train (all three)."""
    return {"name": name, "kind": kind, "dtype": dtype, "batch": batch, "c_in": c_in, "h": hw, "w": hw, "c_out": c_out,
            "k": k, "stride": stride, "pad": pad, "transposed": transposed, "bias": bias, "passes": passes}


def listed():
    return [
        # one projection of an inference request with a few dozen tokens: launches and host path are all there is
        _linear("linear_infer_32", 32, 512, 2048, "f16", "fwd"),
        # the smallest and the largest training shape of the projection sweep (MLP of a transformer block)
        _linear("linear_mlp_4096x512", 4096, 512, 2048, "f16", "train"),
        _linear("linear_mlp_16384x2048", 16384, 2048, 8192, "f16", "train"),
        # the 1000-way head of a classifier in the reference's default precision; the width is no multiple of a tile
        _linear("linear_head_f32", 256, 2048, 1000, "f32", "train"),
        # attention scores Q K^T of 8 heads x 8 sequences at a ragged length, one batched matmul call
        {"name": "matmul_scores_f16", "kind": "matmul", "dtype": "f16", "batch": 64, "m": 333, "kdim": 64, "n": 333},
        # the reference's CPU baseline layer in its own tensors: fp32 NCHW
        _conv("conv3x3_f32_nchw", "conv", "f32", 8, 64, 56, 64, 3, 1, 1),
        # RGB stem: few channels, large image, memory-bound, no input gradient
        _conv("stem7x7_rgb", "conv", "f16", 64, 3, 224, 64, 7, 2, 3, bias=False, passes="fwd+dw"),
        # the 3x3 layer of a residual block at training batch
        _conv("conv3x3_64_b256", "conv", "f16", 256, 64, 56, 64, 3, 1, 1, bias=False),
        # a decoder layer of the U-Net generator (transposed, stride 2, input with the skip concatenated)
        _conv("convT4x4_512_128", "conv", "f16", 64, 512, 32, 128, 4, 2, 1, transposed=True, bias=False),
        # the reference's autocast path, as a program that swaps the extension in calls it
        _conv("dropin_autocast_s2", "dropin", "autocast", 64, 128, 28, 128, 3, 2, 1),
        # the first stage's residual block of the ResNet-50 step at its micro-batch: three convolutions, each with batch
        # norm and ReLU, and the residual add, on tensors larger than L2
        {"name": "bottleneck_56_b256", "kind": "block", "batch": 256, "c_in": 256, "hw": 56, "c_mid": 64, "stride": 1},
        # a training step of the U-Net generator on one GPU's share of a batch of 64 over four, issued call by call
        {"name": "unet_step_b16", "kind": "step", "net": "unet", "batch": 16, "hw": 256, "graph": False},
    ]


# ------------------------------------------------------------------ drawn cases --
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, lo, hi):
    """A channel or feature count: mostly round ones (layers are made so), the rest any."""
    v = _log_int(rng, lo, hi)
    r = rng.random()
    if r < 0.35 and v >= 64:
        return v // 64 * 64
    if r < 0.75 and v >= 8:
        return v // 8 * 8
    return v


# kernel, stride, padding of the layers in use; transposed ones
_CONV_FORMS = [(1, 1, 0), (1, 2, 0), (3, 1, 1), (3, 1, 1), (3, 2, 1), (4, 2, 1), (5, 1, 2), (7, 2, 3)]
_CONVT_FORMS = [(4, 2, 1), (4, 2, 1), (2, 2, 0), (3, 1, 1)]


def draw(rng):
    while True:
        case = _draw_any(rng)
        w = work(case)
        f32 = case.get("dtype") in ("f32", "autocast")
        # no dearer than the largest listed layer / step (fp32 products cost three tensor-core ones at half the rate)
        if w["flops"] <= (2.0e11 if f32 else 1.2e12) and w["bytes"] <= 1.7e9:
            return case


def _draw_any(rng):
    r = rng.random()
    if r < 0.30:
        f16 = rng.random() < 0.7
        c = _linear("", _log_int(rng, 16, 16384), _width(rng, 64, 4096), _width(rng, 64, 8192), "f16" if f16 else "f32",
                    "fwd" if rng.random() < 0.3 else "train")
    elif r < 0.42:
        c = {"name": "", "kind": "matmul", "dtype": rng.choice(["f16", "f16", "f32"]), "batch": _log_int(rng, 1, 128),
             "m": _log_int(rng, 32, 1024), "kdim": rng.choice([32, 64, 64, 96, 128]), "n": _log_int(rng, 32, 1024)}
    elif r < 0.85:
        transposed = rng.random() < 0.3
        k, s, p = rng.choice(_CONVT_FORMS if transposed else _CONV_FORMS)
        rgb = rng.random() < 0.15
        c_in, c_out = _width(rng, 16, 1024), _width(rng, 16, 1024)
        if rgb and transposed:
            c_out, c_in = 3, min(c_in, 256)   # a net's image output
        elif rgb:
            c_in, c_out = 3, min(c_out, 256)  # a net's stem
        hw = _log_int(rng, 4, 224 if rgb and not transposed else 112)
        kind = rng.choice(["conv", "conv", "conv", "conv_f32", "dropin"])
        dtype = {"conv": "f16", "conv_f32": "f32", "dropin": rng.choice(["autocast", "f32"])}[kind]
        c = _conv("", "dropin" if kind == "dropin" else "conv", dtype, _log_int(rng, 1, 256), c_in, hw, c_out, k, s, p,
                  transposed=transposed, bias=rng.random() < 0.5, passes="fwd" if rng.random() < 0.25 else "train")
    elif r < 0.95:
        # a block of one of the four stages: in the middle of a stage, or its first (projection, stride 2)
        stage = rng.randrange(4)
        mid, first = 64 * 2 ** stage, rng.random() < 0.35
        hw = max(7, (224 if rng.random() < 0.5 else _log_int(rng, 112, 288)) // (4 * 2 ** stage))
        c = {"name": "", "kind": "block", "batch": _log_int(rng, 8, 256), "c_mid": mid,
             "c_in": (mid * 2 if stage else 64) if first else mid * 4, "hw": hw * (2 if first and stage else 1),
             "stride": 2 if first and stage else 1}
    else:
        c = {"name": "", "kind": "step", "net": "unet", "batch": _log_int(rng, 12, 32), "hw": 256, "graph": rng.random() < 0.5}
    del c["name"]
    return c


# ------------------------------------------------------------------ state --
_TORCH = {"f16": torch.float16, "f32": torch.float32, "autocast": torch.float32}
_REF = {"f16": _nectarml.DType.Float16, "f32": _nectarml.DType.Float32, "autocast": _nectarml.DType.Float32}


def _geometry(case):
    s, p = case["stride"], case["pad"]
    return ConvGeometry(case["batch"], case["c_in"], case["h"], case["w"], case["c_out"], case["k"], case["k"], (s, s), (p, p),
                        transposed=case["transposed"])


def _conv_out_hw(case):
    k, s, p = case["k"], case["stride"], case["pad"]
    if case["transposed"]:
        return (case["h"] - 1) * s - 2 * p + k, (case["w"] - 1) * s - 2 * p + k
    return (case["h"] + 2 * p - k) // s + 1, (case["w"] + 2 * p - k) // s + 1


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    normal = lambda *shape: torch.randn(shape, device=DEV, generator=gen)  # noqa: E731
    if case["kind"] == "step":
        return _prepare_step(case, seed, gen)
    if case["kind"] == "block":
        return _prepare_block(case, gen)
    dt = _TORCH[case["dtype"]]
    state = {"case": case}
    if case["kind"] == "linear":
        rows, fin, fout = case["rows"], case["fin"], case["fout"]
        bound = math.sqrt(6.0 / (fin + fout))  # Xavier-uniform
        state.update(x=normal(rows, fin).to(dt), w=((torch.rand(fout, fin, device=DEV, generator=gen) * 2 - 1) * bound).to(dt),
                     b=(normal(fout) * 0.1).to(dt), dy=normal(rows, fout).to(dt), math="f16" if case["dtype"] == "f16" else "3xtf32")
    elif case["kind"] == "matmul":
        state.update(a=normal(case["batch"], case["m"], case["kdim"]).to(dt), b=normal(case["batch"], case["kdim"], case["n"]).to(dt))
    else:
        g = _geometry(case)
        nhwc = case["dtype"] == "f16"
        layout = "nhwc" if nhwc else "nchw"
        fan_in = case["c_in"] * case["k"] * case["k"]
        state.update(g=g, layout=layout, out_hw=_conv_out_hw(case), math="f16" if nhwc else "3xtf32",
                     x=normal(*g.act_shape("in", layout)).to(dt), w=(normal(*g.weight_shape()) * math.sqrt(2.0 / fan_in)).to(dt),
                     b=(normal(case["c_out"]) * 0.1).to(dt) if case["bias"] else None, dy=normal(*g.act_shape("out", layout)).to(dt))
    return state


def _prepare_step(case, seed, gen):
    n, hw = case["batch"], case["hw"]
    net, count = train.Pix2PixGenerator(DEV), n * hw * hw * 3
    x, target = ((torch.rand(n, hw, hw, 3, device=DEV, generator=gen) * 2 - 1).half() for _ in range(2))
    net.init(seed=seed)
    step = train.TrainStep(net, "l1", lr=2e-4, momentum=0.9, weight_decay=1e-4)
    state = {"case": case, "net": net, "step": step, "x": x, "target": target, "count": count, "graph": None}
    if case["graph"]:  # the static inputs of the graph are x and target, as a loader would fill them
        state["graph"] = step.capture(x, target, count)[False]
    return state


def _prepare_block(case, gen):
    n, hw, c_in, mid, stride = (case[v] for v in ("batch", "hw", "c_in", "c_mid", "stride"))
    store = train.ParamStore(DEV)
    conv = lambda ci, co, k, s: train.Conv(store, ci, co, k, s, k // 2)  # noqa: E731
    layers = {"c1": conv(c_in, mid, 1, 1), "b1": train.BatchNormAct(store, mid), "c2": conv(mid, mid, 3, stride),
              "b2": train.BatchNormAct(store, mid), "c3": conv(mid, mid * 4, 1, 1), "b3": train.BatchNormAct(store, mid * 4)}
    if c_in != mid * 4:
        layers.update(cd=conv(c_in, mid * 4, 1, stride), bd=train.BatchNormAct(store, mid * 4))
    store.finalize(1)
    for i, shape in enumerate(store.shapes):
        if len(shape) == 4:  # Kaiming-normal
            store.w32(i).copy_(torch.randn(shape, device=DEV, generator=gen) * math.sqrt(2.0 / math.prod(shape[1:])))
    for layer in layers.values():
        if isinstance(layer, train.BatchNormAct):
            layer.gamma.fill_(1.0)
    store.sync_half()
    out = (hw - 1) // stride + 1
    x = torch.randn(n, hw, hw, c_in, device=DEV, generator=gen).relu_().half().requires_grad_()  # the block before ends in a ReLU
    dy = ((torch.rand(n, out, out, mid * 4, device=DEV, generator=gen) * 2 - 1) * 0.1).half()    # gradient of a scaled loss
    return {"case": case, "store": store, "layers": layers, "x": x, "dy": dy,
            "token": torch.zeros((), device=DEV, requires_grad=True)}


# ------------------------------------------------------------------ one pass --
class _Result:
    """A result pointer of the drop-in, owned: what the reference's tensor object is around such a pointer."""

    def __init__(self, ptr, shape, dtype):
        self.ptr, self.n = ptr, math.prod(shape)
        self.dtype = dtype
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f2" if dtype == _nectarml.DType.Float16 else "<f4",
                                         "data": (ptr, False), "version": 2, "strides": None}

    def __del__(self):
        _nectarml.free_cuda(self.ptr, self.n, self.dtype)


def _own(ptr, shape, dtype):
    return torch.as_tensor(_Result(ptr, shape, dtype), device=DEV)


def run(state):
    case = state["case"]
    kind, passes = case["kind"], case.get("passes")
    if kind == "linear":
        x, w, dy, m = state["x"], state["w"], state["dy"], state["math"]
        y = ops.linear_forward(x, w, state["b"], math=m)
        if passes == "fwd":
            return y
        dw, db = ops.linear_backward_weight(x, dy, math=m)
        return y, dw, db, ops.linear_backward_data(dy, w, math=m)
    if kind == "conv":
        g, x, w, dy, lay, m = (state[k] for k in ("g", "x", "w", "dy", "layout", "math"))
        y = ops.conv_forward(g, x, w, state["b"], layout=lay, math=m)
        if passes == "fwd":
            return y
        dw, db = ops.conv_backward_weight(g, x, dy, layout=lay, math=m, want_bias_grad=case["bias"])
        if passes == "fwd+dw":
            return y, dw, db
        return y, dw, db, ops.conv_backward_data(g, dy, w, layout=lay, math=m)
    if kind == "dropin":
        return _run_dropin(state, case, passes)
    if kind == "matmul":
        a, b, dt = state["a"], state["b"], _REF[case["dtype"]]
        return _own(_nectarml.tensor.matmul(a.data_ptr(), b.data_ptr(), a.shape, b.shape, dt), (case["batch"], case["m"], case["n"]), dt)
    if kind == "block":
        return _run_block(state)
    step, store = state["step"], state["net"].store
    if state["graph"] is not None:
        graph, loss = state["graph"]
        graph.replay()
        step.optimizer_step()
    else:
        loss = step([(state["x"], state["target"])], state["count"])
    return {"loss": loss, "grad": store.grad, "params": store.p32, "params_f16": store.p16, "velocity": store.vel,
            "overflow": store.found_inf}


def _run_block(state):
    store, lay, x, t = state["store"], state["layers"], state["x"], state["token"]
    store.begin_backward(last_micro_batch=True)
    idn = lay["bd"](lay["cd"](x, t), t, train.ACT_NONE) if "cd" in lay else x
    y = lay["b1"](lay["c1"](x, t), t, train.ACT_RELU)
    y = lay["b2"](lay["c2"](y, t), t, train.ACT_RELU)
    y = lay["b3"](lay["c3"](y, t), t, train.ACT_RELU, residual=idn)
    (dx,) = torch.autograd.grad(y, (x,), state["dy"])
    store.sgd_step(0.001, 0.9, 1e-4, 1.0 / 16384.0)
    return {"y": y.detach(), "dx": dx, "grad": store.grad, "params": store.p32, "params_f16": store.p16, "velocity": store.vel,
            "overflow": store.found_inf}


def _run_dropin(state, case, passes):
    x, w, b, dy = state["x"], state["w"], state["b"], state["dy"]
    n, ci, h, wd, co, k, s, p = (case[v] for v in ("batch", "c_in", "h", "w", "c_out", "k", "stride", "pad"))
    ho, wo = state["out_hw"]
    dt, f32, half = _REF[case["dtype"]], _nectarml.DType.Float32, case["dtype"] == "autocast"
    conv, tr = _nectarml.tensor.conv, case["transposed"]
    out = (n, co, ho, wo)
    head = (x.data_ptr(), x.numel(), w.data_ptr(), w.numel(), b.data_ptr() if b is not None else 0, co if b is not None else 0,
            math.prod(out), n, ci, h, wd, co, k, k, s, s, p, p, 1, 1)
    ptr = conv.conv_transpose2d(*head, 0, 0, 1, dt, half) if tr else conv.conv2d(*head, 1, dt, half)
    y = _own(ptr, out, dt)
    if passes == "fwd":
        return y
    back = (n, ci, h, wd, co, k, k, ho, wo, s, s, p, p, 1, 1)
    dx = (conv.conv_transpose2d_backward_input if tr else conv.conv2d_backward_input)(dy.data_ptr(), w.data_ptr(), *back, 1, dt)
    dw = (conv.conv_transpose2d_backward_weight if tr else conv.conv2d_backward_weight)(dy.data_ptr(), x.data_ptr(), *back, dt)
    return y, _own(dx, tuple(x.shape), f32), _own(dw, tuple(w.shape), f32)


# ------------------------------------------------------------------ accounting --
def _layer_work(x, w, y, macs, passes, es, es_y=None):
    """Elements of input, weight and output, multiply-adds of one pass -> bytes and operations of the passes: forward
    reads x, w and writes y; the weight gradient reads x, dy and writes dw (fp32); the input gradient reads dy, w and
    writes dx.  What two passes read counts once."""
    by, fl = (x + w + y) * es, 2.0 * macs
    if passes != "fwd":
        by, fl = by + y * es + w * 4, fl + 2.0 * macs
    if passes == "train":
        by, fl = by + x * es, fl + 2.0 * macs
    return {"bytes": float(by), "flops": fl}


def work(case):
    kind = case["kind"]
    es = 2 if case.get("dtype") == "f16" else 4
    if kind == "linear":
        r, i, o = case["rows"], case["fin"], case["fout"]
        return _layer_work(r * i, i * o + o, r * o, r * i * o, case["passes"], es)
    if kind == "matmul":
        n, m, k, c = case["batch"], case["m"], case["kdim"], case["n"]
        return {"bytes": float(n * (m * k + k * c + m * c) * es), "flops": 2.0 * n * m * k * c}
    if kind in ("conv", "dropin"):
        ho, wo = _conv_out_hw(case)
        n, ci, co, kk = case["batch"], case["c_in"], case["c_out"], case["k"] ** 2
        pixels = n * (case["h"] * case["w"] if case["transposed"] else ho * wo)
        return _layer_work(n * ci * case["h"] * case["w"], ci * co * kk, n * co * ho * wo, pixels * ci * co * kk, case["passes"], es)
    n, hw = case["batch"], case["hw"]
    if kind == "block":
        ci, mid, out = case["c_in"], case["c_mid"], (case["hw"] - 1) // case["stride"] + 1
        params, macs = mid * (ci + mid * 13), hw * hw * ci * mid + out * out * mid * mid * 13
        if ci != mid * 4:
            params, macs = params + ci * mid * 4, macs + out * out * ci * mid * 4
        tensors = 2 * n * (hw * hw * ci + out * out * mid * 4)  # x, y and their gradients
    else:
        macs, params = _unet_macs(hw)
        tensors = 2 * n * hw * hw * 3                           # the image and the target
    # parameters and momentum are read and written, gradients and the fp16 copy written
    return {"bytes": float(tensors * 2 + params * (4 * 2 + 4 * 2 + 4 + 2)), "flops": (3 if kind == "block" else 1) * 2.0 * n * macs}


def _unet_macs(hw):
    """Multiply-adds per image of the three passes of every layer (two of the first), and parameters."""
    widths = [64, 128, 256, 512, 512, 512, 512, 512]
    macs, params, side, c = 0, 0, hw, 3
    for i, co in enumerate(widths):
        side //= 2
        macs += (2 if i == 0 else 3) * side ** 2 * c * co * 16
        params, c = params + c * co * 16, co
    for i, co in enumerate(widths[-2::-1] + [3]):
        ci = c if i == 0 else 2 * c
        macs += 3 * side ** 2 * ci * co * 16
        params, side, c = params + ci * co * 16, side * 2, co
    return macs, params


def tolerance(case):
    kind = case["kind"]
    if kind in ("block", "step"):
        # fp16 activations: a value that rounds the other way can flip a ReLU behind it, and each flip is a jump in the
        # gradients in front of it.  Evaluations that differ in rounding alone show 1e-2 of the gradient (more after a
        # further step), and single small gradients of the first layers by as much as they are.
        return {"rel": 2e-2, "max": 0.99}
    if case["dtype"] == "f32":
        # 3xTF32: fp32 sums.  The tensor core drops the low bits at each step of a sum, so it is off by 2.5e-9 of itself per
        # term (measured against float64); a weight gradient is summed in shares.
        if kind == "linear":
            terms = max(case["fin"], case["fout"], min(case["rows"], 8192))
        elif kind == "matmul":
            terms = case["kdim"]
        else:
            ho, wo = _conv_out_hw(case)
            terms = max(max(case["c_in"], case["c_out"]) * case["k"] ** 2, min(case["batch"] * max(ho * wo, case["h"] * case["w"]), 8192))
        return {"rel": max(1e-5, 2.5e-9 * terms)}
    return {"rel": 1e-3}  # results or operands rounded to fp16 (half an ulp is 5e-4), fp32 sums
