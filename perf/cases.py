"""Workloads of the analog layers, each with its inputs, one pass through the public modules, the work it
cannot do without and the tolerance of its results.

Kinds of case:

* ``linear`` -- one ``AnalogLinear``: evaluation forward, or a training forward + backward.
* ``mlp``    -- the gated MLP of a decoder layer (``AnalogLinear`` gate / up projection, ``swiglu``,
  ``AnalogLinear`` down projection).
* ``conv``   -- one 3 x 3 ``AnalogConv2d`` of a CIFAR-shaped ResNet, training forward + backward.
"""
import os
import sys

import torch

_PACKAGE_DIR = os.path.abspath("aihwkit-lightning_b200")
if _PACKAGE_DIR not in sys.path:
    sys.path.insert(0, _PACKAGE_DIR)

from aihwkit_lightning_b200.nn import AnalogConv2d, AnalogLinear  # noqa: E402
from aihwkit_lightning_b200.nn.decoder_ops import swiglu  # noqa: E402
from aihwkit_lightning_b200.simulator.configs import TorchInferenceRPUConfig  # noqa: E402
from aihwkit_lightning_b200.simulator.enums import WeightNoiseInjectionType, WeightQuantizationType  # noqa: E402

DEVICE = "cuda"
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}


def _linear(rows, k, n, tile, dtype="bf16", train=False, dynamic=True, adc=True, out_noise=0.0, w_noise=0.0,
            discretize=False, bias=False):
    return dict(kind="linear", rows=rows, k=k, n=n, tile=tile, dtype=dtype, train=train, dynamic=dynamic, adc=adc,
                out_noise=out_noise, w_noise=w_noise, discretize=discretize, bias=bias)


def _mlp(rows, d, hidden, train):
    return dict(kind="mlp", rows=rows, d=d, hidden=hidden, tile=512, dtype="bf16", train=train)


def _conv(batch, cin, cout, size, stride):
    return dict(kind="conv", batch=batch, cin=cin, cout=cout, size=size, stride=stride, tile=256, dtype="f32")


def listed():
    return [
        # decoding, one token through one layer: the smallest call, where latency counts
        dict(_linear(1, 2048, 2048, 512), name="decode_1x2048"),
        # decoding, a batch of 16 sequences through the gated MLP of a decoder layer (d = 3072, MLP 8192)
        dict(_mlp(16, 3072, 8192, False), name="decode_mlp_16"),
        # a short prompt: a few hundred rows against a layer of ordinary size
        dict(_linear(256, 4096, 4096, 512), name="prefill_256x4096"),
        # a long prompt, wide tiles
        dict(_linear(4096, 8192, 8192, 1024), name="prefill_4096x8192"),
        # evaluation of a layer whose sizes divide by nothing (tiles of 500, 777 outputs)
        dict(_linear(333, 1000, 777, 512, bias=True), name="eval_ragged_333"),
        # hardware-aware training of one layer: per-token ranges, DAC, ADC, output and weight noise
        dict(_linear(8192, 4096, 4096, 512, train=True, out_noise=0.04, w_noise=0.02), name="train_8192x4096"),
        # the same on ragged sizes (tiles of 500, rows and outputs that fill no block)
        dict(_linear(1000, 2500, 1500, 512, train=True, out_noise=0.04, w_noise=0.02, bias=True), name="train_ragged_1000"),
        # fp32 training with learned static ranges: a small layer, then one where the products bound the step
        dict(_linear(512, 1024, 1024, 512, "f32", True, False, False, 0.04, 0.02, bias=True), name="train_f32_512x1024"),
        dict(_linear(4096, 4096, 4096, 512, "f32", True, False, False, 0.04, 0.02, bias=True), name="train_f32_4096x4096"),
        # ResNet-32 at batch 256: a convolution of the first stage and one of the last
        dict(_conv(256, 16, 16, 32, 1), name="conv_16x32x32"),
        dict(_conv(256, 64, 64, 8, 1), name="conv_64x8x8"),
        # decoder training, 8192 tokens through the gated MLP (no ADC): the largest
        dict(_mlp(8192, 3072, 8192, True), name="train_mlp_8192"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))


def _size(rng, lo, hi, ragged):
    """A size of the range, spread over its logarithm: a multiple of 64, or any number."""
    v = _log_int(rng, lo, hi)
    return v if ragged else max(lo, v // 64 * 64)


def draw(rng):
    kind = rng.choice(["decode", "prefill", "prefill", "train", "train", "train_f32", "conv", "mlp"])
    if kind == "mlp":
        train = rng.random() < 0.5
        return _mlp(_log_int(rng, 128, 8192) if train else _log_int(rng, 1, 64), _size(rng, 512, 3072, False),
                    _size(rng, 1024, 8192, False), train)
    if kind == "conv":
        cin, cout, size, stride = rng.choice([(16, 16, 32, 1), (16, 32, 32, 2), (32, 32, 16, 1), (32, 64, 16, 2), (64, 64, 8, 1)])
        return _conv(_log_int(rng, 16, 256), cin, cout, size, stride)
    ragged = rng.random() < 1 / 3
    tile = rng.choice([256, 512, 1024])
    if kind == "train_f32":
        c = _linear(_log_int(rng, 64, 4096), _size(rng, 256, 4096, ragged), _size(rng, 256, 4096, ragged), tile, "f32", True,
                    rng.random() < 0.5, False, 0.04, 0.02, bias=True)
        limit = 8e10 if ragged else 4.2e11
    elif kind == "train":
        adc = rng.random() < 0.6
        c = _linear(_log_int(rng, 64, 8192), _size(rng, 256, 8192, ragged), _size(rng, 256, 8192, ragged), tile, "bf16", True,
                    rng.random() < 0.6, adc, 0.04, 0.02, rng.random() < 0.3, rng.random() < 0.5)
        limit = 8e10 if ragged else 1e12
    elif kind == "decode":
        c = _linear(_log_int(rng, 1, 64), _size(rng, 512, 16384, ragged), _size(rng, 512, 16384, ragged), tile,
                    adc=rng.random() < 0.7, bias=rng.random() < 0.5)
        limit = 1e10 if ragged else 1e12
    else:
        c = _linear(_log_int(rng, 32, 16384), _size(rng, 512, 8192, ragged), _size(rng, 512, 8192, ragged), tile,
                    adc=rng.random() < 0.7, bias=rng.random() < 0.5)
        limit = 8e10 if ragged else 1e12
    while work(c)["flops"] > limit:  # no more work than the largest case above
        name = max(("rows", "k", "n"), key=lambda f: c[f])
        c[name] = c[name] // 2 if ragged else max(64, c[name] // 2 // 64 * 64)
    return c


def _rpu_config(c):
    rpu = TorchInferenceRPUConfig()
    rpu.mapping.max_input_size = c["tile"]
    rpu.forward.inp_res = 254.0
    if c.get("adc", False):
        rpu.forward.out_res = 254.0
        rpu.forward.out_bound = 10.0
    train = c.get("train", True)
    rpu.forward.out_noise = c.get("out_noise", {"mlp": 0.04, "conv": 0.02}.get(c["kind"], 0.0)) if train else 0.0
    irp = rpu.pre_post.input_range
    irp.enable = True
    irp.dynamic = c.get("dynamic", True)
    if not irp.dynamic:
        irp.learn_input_range = True
        irp.init_value = 3.0
        irp.init_from_data = 0
    w_noise = c.get("w_noise", 0.02)
    if train and w_noise > 0:
        rpu.modifier.noise_type = WeightNoiseInjectionType.ADD_NORMAL_PER_CHANNEL
        rpu.modifier.std_dev = w_noise
    if c.get("discretize", False):
        rpu.modifier.quantization_type = WeightQuantizationType.DISCRETIZE_PER_CHANNEL
        rpu.modifier.res = 254.0
    return rpu


def _module(c):
    rpu = _rpu_config(c)
    opts = dict(rpu_config=rpu, device=DEVICE, dtype=DTYPES[c["dtype"]])
    if c["kind"] == "linear":
        layers = [AnalogLinear(c["k"], c["n"], bias=c["bias"], **opts)]
    elif c["kind"] == "mlp":
        layers = [AnalogLinear(c["d"], 2 * c["hidden"], bias=False, **opts),
                  AnalogLinear(c["hidden"], c["d"], bias=False, **opts)]
    else:
        layers = [AnalogConv2d(c["cin"], c["cout"], 3, stride=c["stride"], padding=1, bias=False, **opts)]
    for layer in layers:
        layer.train(c.get("train", True))
    return torch.nn.ModuleList(layers)


def prepare(case, seed):
    """The layers and the activations (and output gradients) of one pass; the noise of a training pass comes from
    torch's generator, seeded last."""
    torch.manual_seed(seed)
    layers = _module(case)
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    dtype = DTYPES[case["dtype"]]
    if case["kind"] == "conv":
        shape = (case["batch"], case["cin"], case["size"], case["size"])
        out_size = (case["size"] - 1) // case["stride"] + 1
        out_shape = (case["batch"], case["cout"], out_size, out_size)
    else:
        shape = (case["rows"], case["k"] if case["kind"] == "linear" else case["d"])
        out_shape = (case["rows"], case["n"] if case["kind"] == "linear" else case["d"])
    train = case.get("train", True)
    x = torch.randn(shape, device=DEVICE, generator=gen, dtype=torch.float32).to(dtype)
    if case["kind"] == "conv":
        x.relu_()  # the activations of a ResNet block
    g = torch.randn(out_shape, device=DEVICE, generator=gen, dtype=torch.float32).to(dtype) if train else None
    torch.cuda.manual_seed(seed)
    return dict(kind=case["kind"], train=train, layers=layers, x=x.requires_grad_(train), g=g)


def _forward(state):
    layers, x = state["layers"], state["x"]
    if state["kind"] == "mlp":
        return layers[1](swiglu(layers[0](x)))
    return layers[0](x)


def run(state):
    if not state["train"]:
        with torch.no_grad():
            return _forward(state)
    params = list(state["layers"].parameters())
    state["x"].grad = None
    for p in params:
        p.grad = None
    out = _forward(state)
    out.backward(state["g"])
    return [out.detach(), state["x"].grad] + [p.grad for p in params if p.grad is not None]


def _layer_work(rows, k, n, es, train):
    flops = 2.0 * rows * k * n
    inputs, weights, outputs = rows * k * es, n * k * es, rows * n * es
    if not train:
        return inputs + weights + outputs, flops
    # read x, w, the output's gradient; write the output and both gradients
    return 2 * inputs + 2 * weights + 2 * outputs, 3 * flops


def work(case):
    es = 2 if case["dtype"] == "bf16" else 4
    train = case.get("train", True)
    if case["kind"] == "linear":
        b, f = _layer_work(case["rows"], case["k"], case["n"], es, train)
        return {"bytes": b, "flops": f}
    if case["kind"] == "mlp":
        rows, d, hidden = case["rows"], case["d"], case["hidden"]
        b1, f1 = _layer_work(rows, d, 2 * hidden, es, train)
        b2, f2 = _layer_work(rows, hidden, d, es, train)
        return {"bytes": b1 + b2, "flops": f1 + f2}
    out_size = (case["size"] - 1) // case["stride"] + 1
    k = 9 * case["cin"]
    pixels_in, pixels_out = case["batch"] * case["size"] ** 2, case["batch"] * out_size ** 2
    return {"bytes": es * 2 * (pixels_in * case["cin"] + pixels_out * case["cout"] + case["cout"] * k),
            "flops": 6.0 * pixels_out * case["cout"] * k}


def tolerance(case):
    # bf16: results are rounded to 8 significant bits after every step of the output stage, and sums in another order
    # move a share of the converter's codes by one level.  Keeping the output stage in fp32 instead changes the
    # results of an evaluation by 7e-3 .. 9e-3.
    if case["dtype"] == "bf16":
        return {"rel": 1e-2}
    # fp32 sums in another order, operands split into bf16 planes on the tensor cores: 6e-6 between the two engines
    return {"rel": 2e-5}
