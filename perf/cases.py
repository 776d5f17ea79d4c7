"""Performance cases: the work that a user of this framework has it do, through
its public entry points (`raw_ops`, `optimizers`).

A case is a plain dict.  `prepare` makes what a program has in hand before the
call (device tensors, an optimizer), `run` is one pass as the program makes it,
`work` what such a pass cannot do without, `tolerance` how far two correct
implementations of the same precision may lie apart.

Ops:
  bn_train       FusedBatchNormV3 (training) and FusedBatchNormGradV3 of one layer
  bn_resnet50    the same for one layer of each of the nine shapes that ResNet-50's
                 BatchNorm layers have (all forwards, then the gradients in reverse
                 order, as a training step meets them)
  bn_resnet50_infer  FusedBatchNormV3 with is_training=False for those nine shapes
  bias_relu      MusaBiasAddRelu, then MusaBiasAddReluGrad
  bias_swish     MusaBiasAddSwish
  adam           ResourceApplyAdam on one flat parameter vector
  adam_block     MusaAdam.apply_gradients over the 16 variables of one transformer
                 encoder block (fp32 variables, fp32 or bf16 gradients)
  layer_norm     MusaLayerNorm, then MusaLayerNormGrad
  rms_norm       MusaRmsNorm, then MusaRmsNormGradDx
"""
import math

import torch

from tensorflow_musa_extension_b200 import optimizers, raw_ops

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
EPS = 1e-3
# Height, width and channels of ResNet-50's BatchNorm layers at 224 x 224.
RESNET50 = ((112, 112, 64), (56, 56, 64), (56, 56, 256), (28, 28, 128), (28, 28, 512),
            (14, 14, 256), (14, 14, 1024), (7, 7, 512), (7, 7, 2048))
RESNET50_VALUES = sum(h * w * c for h, w, c in RESNET50)   # per image
# lr, beta1, beta2, epsilon and the two powers of a tenth step.
LR, BETA1, BETA2, ADAM_EPS = 1e-3, 0.9, 0.999, 1e-7
POWERS = (BETA1 ** 10, BETA2 ** 10)
# The most that a drawn case works on: values of one activation tensor, parameters.
MAX_VALUES = 1 << 27
MAX_PARAMS = 1 << 26


def listed():
    return [
        # The smallest layers (a small image or a small batch): launches and
        # host work decide.
        {"name": "bn_f32_8x14x14x64", "op": "bn_train", "dtype": "f32", "layout": "NHWC",
         "n": 8, "h": 14, "w": 14, "c": 64, "factor": 1.0},
        # An ordinary fp32 layer, running averages blended in the same call.
        {"name": "bn_f32_32x56x56x64", "op": "bn_train", "dtype": "f32", "layout": "NHWC",
         "n": 32, "h": 56, "w": 56, "c": 64, "factor": 0.1},
        # A large half-precision layer.
        {"name": "bn_f16_256x28x28x256", "op": "bn_train", "dtype": "f16", "layout": "NHWC",
         "n": 256, "h": 28, "w": 28, "c": 256, "factor": 1.0},
        # Channels first (models that were written for that layout), planes of
        # 7 x 7: no plane is a whole number of vector accesses.
        {"name": "bn_nchw_bf16_64x512x7x7", "op": "bn_train", "dtype": "bf16", "layout": "NCHW",
         "n": 64, "h": 7, "w": 7, "c": 512, "factor": 1.0},
        # Training ResNet-50: a small batch (fine-tuning, many replicas) and the
        # full batch of one GPU.
        {"name": "bn_resnet50_bf16_b32", "op": "bn_resnet50", "dtype": "bf16", "batch": 32},
        {"name": "bn_resnet50_bf16_b256", "op": "bn_resnet50", "dtype": "bf16", "batch": 256},
        # Serving ResNet-50 with a batch of eight.
        {"name": "bn_resnet50_infer_bf16_b8", "op": "bn_resnet50_infer", "dtype": "bf16",
         "batch": 8},
        # A dense layer's epilogue and its backward, full size.
        {"name": "bias_relu_f16_65536x1024", "op": "bias_relu", "dtype": "f16",
         "rows": 65536, "c": 1024},
        # An odd width (a thousand classes and background): no row starts on a
        # vector boundary.
        {"name": "bias_swish_f32_4096x1001", "op": "bias_swish", "dtype": "f32",
         "rows": 4096, "c": 1001},
        # The optimizer step of ResNet-50 as one flat vector.
        {"name": "adam_f32_25557032", "op": "adam", "dtype": "f32", "params": 25557032},
        # The optimizer step of one encoder block, variable by variable.
        {"name": "adam_block_bf16_768", "op": "adam_block", "dtype": "bf16", "width": 768},
        # Layer normalisation between the blocks: 8 sequences of 2048.
        {"name": "layer_norm_bf16_16384x1024", "op": "layer_norm", "dtype": "bf16",
         "rows": 16384, "c": 1024},
    ]


def _log(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _width(rng, lo, hi):
    """A channel count: mostly a multiple of 32, the others as they fall."""
    c = _log(rng, lo, hi)
    return max(32, c // 32 * 32) if rng.random() < 0.7 else c


def draw(rng):
    op = rng.choice(("bn_train", "bn_train", "bn_train", "bn_resnet50", "bn_resnet50_infer",
                     "bias_relu", "bias_swish", "adam", "adam_block", "layer_norm", "rms_norm"))
    case = {"op": op, "dtype": rng.choice(tuple(DTYPES))}
    if op == "bn_train":
        case["layout"] = rng.choice(("NHWC", "NHWC", "NCHW"))
        case["h"] = case["w"] = rng.choice((1, 7, 14, 28, 56, 112, _log(rng, 2, 112)))
        case["c"] = _width(rng, 16, 2048)
        most = MAX_VALUES // (case["h"] * case["w"] * case["c"])
        case["n"] = _log(rng, 2, max(2, min(most, 65536 if case["h"] == 1 else 256)))
        case["factor"] = rng.choice((1.0, 0.1))
    elif op == "bn_resnet50":
        case["batch"] = _log(rng, 2, 256)
        case["dtype"] = rng.choice(("bf16", "f16"))
    elif op == "bn_resnet50_infer":
        case["batch"] = _log(rng, 1, 256)
    elif op == "adam":
        case["params"] = _log(rng, 1000, MAX_PARAMS)
        case["dtype"] = rng.choice(("f32", "bf16"))   # fp16 cannot hold second moments
    elif op == "adam_block":
        case["width"] = _log(rng, 64, 2048)
        case["dtype"] = rng.choice(("f32", "bf16"))
    else:
        if op == "rms_norm":
            case["dtype"] = rng.choice(("f32", "bf16"))
        case["c"] = _width(rng, 64, 8192)
        case["rows"] = _log(rng, 16, min(131072, MAX_VALUES // case["c"]))
    return case


# ------------------------------------------------------------------ inputs --

class _Inputs:
    """Device tensors drawn from one seed."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)

    def normal(self, shape, std, mean=0.0, dtype=torch.float32):
        t = torch.empty(shape, dtype=torch.float32, device="cuda")
        return t.normal_(mean, std, generator=self.gen).to(dtype)

    def uniform(self, shape, lo, hi, dtype=torch.float32):
        t = torch.empty(shape, dtype=torch.float32, device="cuda")
        return t.uniform_(lo, hi, generator=self.gen).to(dtype)

    def batch_norm(self, shape, c, dtype):
        return {"x": self.normal(shape, 3.0, 1.0, dtype), "dy": self.normal(shape, 1e-2, 0.0, dtype),
                "scale": self.uniform((c,), 0.5, 1.5), "offset": self.normal((c,), 0.1),
                "mean": self.normal((c,), 0.1, 1.0), "variance": self.uniform((c,), 8.0, 10.0)}


def _block_shapes(d):
    """The 16 variables of an encoder block of width d: four attention
    projections, two dense layers, two normalisations."""
    shapes = [(d, d), (d,)] * 4 + [(d, 4 * d), (4 * d,), (4 * d, d), (d,)] + [(d,), (d,)] * 2
    assert len(shapes) == 16
    return shapes


def prepare(case, seed):
    r = _Inputs(seed)
    op, dtype = case["op"], DTYPES[case["dtype"]]
    s = {"case": case}
    if op == "bn_train":
        n, h, w, c = (case[k] for k in "nhwc")
        shape = (n, h, w, c) if case["layout"] == "NHWC" else (n, c, h, w)
        s.update(r.batch_norm(shape, c, dtype))
        if case["factor"] == 1.0:   # nothing to blend with: empty inputs, as TensorFlow passes them
            s["mean"] = s["variance"] = torch.empty(0, device="cuda")
    elif op in ("bn_resnet50", "bn_resnet50_infer"):
        s["empty"] = torch.empty(0, device="cuda")
        s["layers"] = []
        for h, w, c in RESNET50:
            layer = r.batch_norm((case["batch"], h, w, c), c, dtype)
            if op == "bn_resnet50_infer":
                del layer["dy"]
            s["layers"].append(layer)
    elif op in ("bias_relu", "bias_swish"):
        shape = (case["rows"], case["c"])
        s["x"] = r.normal(shape, 1.0, 0.0, dtype)
        s["bias"] = r.normal((case["c"],), 0.1, 0.0, dtype)
        if op == "bias_relu":
            s["dy"] = r.normal(shape, 1e-2, 0.0, dtype)
    elif op == "adam":
        n = case["params"]
        s["var"] = r.normal((n,), 0.05, 0.0, dtype)
        s["m"] = r.normal((n,), 1e-4, 0.0, dtype)
        s["v"] = r.uniform((n,), 0.0, 1e-6, dtype)
        s["grad"] = r.normal((n,), 1e-3, 0.0, dtype)
    elif op == "adam_block":
        opt = optimizers.MusaAdam(LR, BETA1, BETA2, ADAM_EPS)
        s["vars"] = [r.normal(shape, 0.05) for shape in _block_shapes(case["width"])]
        s["grads"] = [r.normal(t.shape, 1e-3, 0.0, dtype) for t in s["vars"]]
        # A training run in its tenth step.
        opt.iterations = 10
        for t in s["vars"]:
            opt.get_slot(t, "m").normal_(0.0, 1e-4, generator=r.gen)
            opt.get_slot(t, "v").uniform_(0.0, 1e-6, generator=r.gen)
        s["opt"] = opt
    else:
        shape, c = (case["rows"], case["c"]), case["c"]
        s["x"] = r.normal(shape, 1.0, 0.2, dtype)
        s["dy"] = r.normal(shape, 1e-2, 0.0, dtype)
        s["gamma"] = r.uniform((c,), 0.5, 1.5, dtype)
        s["beta"] = r.normal((c,), 0.1, 0.0, dtype)
    return s


# -------------------------------------------------------------- one pass --

def _resnet50_step(s):
    out = [None] * len(s["layers"])
    for i, p in enumerate(s["layers"]):
        out[i] = raw_ops.FusedBatchNormV3(p["x"], p["scale"], p["offset"], s["empty"], s["empty"],
                                          epsilon=EPS)
    for i in reversed(range(len(out))):
        p, f = s["layers"][i], out[i]
        g = raw_ops.FusedBatchNormGradV3(p["dy"], p["x"], p["scale"], f.reserve_space_1,
                                         f.reserve_space_2, f.reserve_space_3, epsilon=EPS)
        out[i] = (f.y, f.batch_mean, f.batch_variance, g.x_backprop, g.scale_backprop,
                  g.offset_backprop)
    return out


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "bn_train":
        f = raw_ops.FusedBatchNormV3(s["x"], s["scale"], s["offset"], s["mean"], s["variance"],
                                     epsilon=EPS, exponential_avg_factor=case["factor"],
                                     data_format=case["layout"])
        g = raw_ops.FusedBatchNormGradV3(s["dy"], s["x"], s["scale"], f.reserve_space_1,
                                         f.reserve_space_2, f.reserve_space_3, epsilon=EPS,
                                         data_format=case["layout"])
        return tuple(f) + tuple(g)
    if op == "bn_resnet50":
        return _resnet50_step(s)
    if op == "bn_resnet50_infer":
        return [raw_ops.FusedBatchNormV3(p["x"], p["scale"], p["offset"], p["mean"], p["variance"],
                                         epsilon=EPS, is_training=False).y for p in s["layers"]]
    if op == "bias_relu":
        y = raw_ops.MusaBiasAddRelu(s["x"], s["bias"])
        return (y,) + tuple(raw_ops.MusaBiasAddReluGrad(s["dy"], y))
    if op == "bias_swish":
        return raw_ops.MusaBiasAddSwish(s["x"], s["bias"])
    if op == "adam":
        raw_ops.ResourceApplyAdam(s["var"], s["m"], s["v"], POWERS[0], POWERS[1], LR, BETA1, BETA2,
                                  ADAM_EPS, s["grad"])
        return s["var"], s["m"], s["v"]
    if op == "adam_block":
        opt = s["opt"]
        opt.apply_gradients(list(zip(s["grads"], s["vars"])))
        return [(t, opt.get_slot(t, "m"), opt.get_slot(t, "v")) for t in s["vars"]]
    if op == "layer_norm":
        y = raw_ops.MusaLayerNorm(s["x"], s["gamma"], s["beta"])
        return (y,) + tuple(raw_ops.MusaLayerNormGrad(s["dy"], s["x"], s["gamma"], s["beta"]))
    f = raw_ops.MusaRmsNorm(s["x"], s["gamma"])
    return tuple(f) + (raw_ops.MusaRmsNormGradDx(s["x"], f.inv_rms, s["gamma"], s["dy"]),)


# ---------------------------------------------------- what a pass has to do --

def work(case):
    """Bytes: every input once, every output once (a tensor that both halves of
    a pass need counts in each half).  Flops: the arithmetic of the formulas."""
    op, size = case["op"], DTYPES[case["dtype"]].itemsize
    if op == "bn_train":
        values, c = case["n"] * case["h"] * case["w"] * case["c"], case["c"]
        return {"bytes": 5 * size * values + 12 * 4 * c, "flops": 14 * values}
    if op == "bn_resnet50":
        values = case["batch"] * RESNET50_VALUES
        return {"bytes": 5 * size * values, "flops": 14 * values}
    if op == "bn_resnet50_infer":
        values = case["batch"] * RESNET50_VALUES
        return {"bytes": 2 * size * values, "flops": 2 * values}
    if op == "adam":
        n = case["params"]
        return {"bytes": 7 * size * n, "flops": 12 * n}
    if op == "adam_block":
        n = sum(math.prod(shape) for shape in _block_shapes(case["width"]))
        return {"bytes": (6 * 4 + size) * n, "flops": 12 * n}
    values = case["rows"] * case["c"]
    tensors, flops = {"bias_relu": (5, 5), "bias_swish": (2, 5), "layer_norm": (5, 22),
                      "rms_norm": (6, 11)}[op]
    return {"bytes": tensors * size * values, "flops": flops * values}


def tolerance(case):
    """About four times what the path differs from the same formulas in 64 bits
    (2-norms; `max`: single values).  Seen: fp32 element-wise results 7e-8 and
    2e-7, fp32 results of sums 2e-7 and 5e-7 (statistics of large layers 3e-6);
    rounding to fp16 2.1e-4 (swish 2.8e-4) and 5e-4 (8.5e-4), to bf16 1.7e-3
    (2.3e-3) and 3.9e-3 (6.9e-3)."""
    if case["op"] == "adam_block" or (case["op"] == "adam" and case["dtype"] == "f32"):
        return {"rel": 3e-7, "max": 1e-6}
    if case["dtype"] == "f32":
        if case["op"] in ("bias_swish", "bn_resnet50_infer"):
            return {"rel": 3e-7, "max": 2e-6}
        return {"rel": 1e-5, "max": 2e-5}
    return {"f16": {"rel": 1.2e-3, "max": 4e-3}, "bf16": {"rel": 1e-2, "max": 3e-2}}[case["dtype"]]
