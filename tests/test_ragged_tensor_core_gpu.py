"""bf16 layers whose sizes are no multiples of 8 on the tensor cores, against the oracle and the CUDA-core GEMMs of the same
layer: the operands of the two (DAC output, modified weights, noise included) are the same bits, laid out differently."""
import pytest
import torch

import cases as C
from test_parity_gpu import check_close
from util import oracle_run, rel_fro, run_product_layer

pytestmark = pytest.mark.gpu

# One bf16 rounding per tile and per partial sum separates two orders of the same fp32 sum (2^-9 relative each), and
# a share of the ADC codes moves by one level: the bar of every other bf16 comparison of this repository.
BF16_REL = 1e-2

SHAPES = [
    # rows, K, N, tile: what is at the edge
    (333, 1000, 777, 512),    # tiles of 500, odd N
    (65, 2049, 513, 512),     # uneven tiles (410 and 409), one row and one column beyond a block
    (128, 2048, 130, 256),    # K aligned: the pitched layout is the dense one
    (200, 777, 512, -1),      # one tile of 777, N aligned
    (32, 4100, 1030, -1),     # a tile wider than a warp keeps in registers
    (1000, 2500, 1500, 512),
    (300, 1001, 67, 77),      # 13 narrow tiles of 77, few channels
    (8193, 515, 130, 260),    # sums over the rows in two chunks, 64- and 128-column blocks
    (24577, 1000, 777, 512),  # in four
    (1, 70, 9, 35),           # the smallest calls: one row, a few channels, tiles narrower than a k-step
]
OPTIONS = {
    "train": dict(dynamic=True, adc=True, noise=True, discretize=False, learn_clip=False),
    "no_adc": dict(dynamic=True, adc=False, noise=True, discretize=False, learn_clip=False),
    "static_discretize": dict(dynamic=False, adc=True, noise=True, discretize=True, learn_clip=False),
    "plain": dict(dynamic=False, adc=False, noise=False, discretize=False, learn_clip=False),
    "learn_clip": dict(dynamic=True, adc=True, noise=False, discretize=False, learn_clip=True),
}


def _layer(k, n, tile, o):
    from aihwkit_lightning_b200.nn import AnalogLinear
    from aihwkit_lightning_b200.simulator.configs import TorchInferenceRPUConfig
    from aihwkit_lightning_b200.simulator.enums import (WeightClipType, WeightNoiseInjectionType,
                                                        WeightQuantizationType)

    rpu = TorchInferenceRPUConfig()
    rpu.mapping.max_input_size = tile
    rpu.forward.inp_res = 254.0
    if o["adc"]:
        rpu.forward.out_res, rpu.forward.out_bound = 254.0, 10.0
    irp = rpu.pre_post.input_range
    irp.enable, irp.dynamic = True, o["dynamic"]
    if not o["dynamic"]:
        irp.learn_input_range, irp.init_value, irp.init_from_data = True, 2.5, 0
    if o["noise"]:
        rpu.forward.out_noise = 0.04
        rpu.modifier.noise_type, rpu.modifier.std_dev = WeightNoiseInjectionType.ADD_NORMAL_PER_CHANNEL, 0.02
    if o["discretize"]:
        rpu.modifier.quantization_type, rpu.modifier.res = WeightQuantizationType.DISCRETIZE_PER_CHANNEL, 254.0
    if o["learn_clip"]:
        rpu.clip.type = WeightClipType.LEARNABLE_PER_CHANNEL
    torch.manual_seed(3)
    return AnalogLinear(k, n, bias=True, rpu_config=rpu, device="cuda", dtype=torch.bfloat16)


def _pass(layer, x, g, engine):
    from aihwkit_lightning_b200.nn import functional as F

    x = x.detach().clone().requires_grad_(True)
    layer.zero_grad()
    torch.cuda.manual_seed(11)
    with F.operator_settings(engine=engine):
        out = layer(x)
        node = out.grad_fn
        while not hasattr(node, "saved_tensors") or len(node.saved_tensors) < 9:  # the layer's own node
            node = node.next_functions[0][0]
        xq, w_mod = node.saved_tensors[1:3]
        out.backward(g)
    return out.detach(), x.grad, {n: p.grad for n, p in layer.named_parameters() if p.grad is not None}, xq, w_mod


def _dense(t, in_sizes):
    """The tiles of a pitched operand side by side; its padding must be zero."""
    pitch = t.shape[1] // len(in_sizes)
    parts = t.view(t.shape[0], len(in_sizes), pitch)
    for i, width in enumerate(in_sizes):
        assert not parts[:, i, width:].any()
    return torch.cat([parts[:, i, :width] for i, width in enumerate(in_sizes)], dim=1)


@pytest.mark.parametrize("name", OPTIONS)
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_ragged_layer_matches_cuda_cores(shape, name):
    rows, k, n, tile = shape
    layer = _layer(k, n, tile, OPTIONS[name])
    layer.train()
    gen = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(rows, k, device="cuda", generator=gen, dtype=torch.float32).bfloat16()
    g = torch.randn(rows, n, device="cuda", generator=gen, dtype=torch.float32).bfloat16()
    out, gx, grads, xq, w_mod = _pass(layer, x, g, "auto")
    out_s, gx_s, grads_s, xq_s, w_mod_s = _pass(layer, x, g, "simt")
    torch.cuda.synchronize()
    assert (xq.shape[1] != k) == (k % 8 != 0 or any(w % 8 for w in layer.in_sizes))  # the pitched route was taken
    assert torch.equal(_dense(xq, layer.in_sizes), xq_s)
    assert torch.equal(_dense(w_mod, layer.in_sizes), w_mod_s)
    assert rel_fro(out, out_s) <= BF16_REL
    assert rel_fro(gx, gx_s) <= BF16_REL
    assert grads.keys() == grads_s.keys()
    for key in grads:
        assert rel_fro(grads[key], grads_s[key]) <= BF16_REL, key
    layer.eval()
    with torch.no_grad():
        from aihwkit_lightning_b200.nn import functional as F

        ev = layer(x)
        with F.operator_settings(engine="simt"):
            ev_s = layer(x)
    assert rel_fro(ev, ev_s) <= BF16_REL


def test_ragged_layer_unaligned_inputs_and_gradients():
    """Views that start two bytes into an allocation: the sources of the pitched layout have no alignment."""
    rows, k, n = 130, 1001, 515
    layer = _layer(k, n, 512, OPTIONS["train"])
    layer.train()
    x = torch.randn(rows * k + 1, device="cuda").bfloat16()[1:].view(rows, k)
    g = torch.randn(rows * n + 1, device="cuda").bfloat16()[1:].view(rows, n)
    a, b = _pass(layer, x, g, "auto"), _pass(layer, x, g, "simt")
    assert rel_fro(a[0], b[0]) <= BF16_REL and rel_fro(a[1], b[1]) <= BF16_REL
    assert rel_fro(a[2]["weight"], b[2]["weight"]) <= BF16_REL


@pytest.mark.parametrize("name", OPTIONS)
@pytest.mark.parametrize("k,n,tile", [(1000, 777, 512), (1001, 515, 77), (1024, 131, 512)])
def test_ragged_layer_unaligned_weights(k, n, tile, name):
    """Weights two bytes into an allocation: the same modified weights, noise included, as the dense pass writes."""
    rows = 70
    layer = _layer(k, n, tile, OPTIONS[name])
    layer.train()
    flat = torch.empty(n * k + 1, device="cuda", dtype=torch.bfloat16)
    view = flat[1:].view(n, k)
    view.copy_(layer.weight.data)
    layer.weight.data = view
    x, g = torch.randn(rows, k, device="cuda").bfloat16(), torch.randn(rows, n, device="cuda").bfloat16()
    out, gx, grads, xq, w_mod = _pass(layer, x, g, "auto")
    out_s, gx_s, grads_s, xq_s, w_mod_s = _pass(layer, x, g, "simt")
    assert (xq.shape[1] != k) == any(w % 8 for w in layer.in_sizes)
    assert torch.equal(_dense(xq, layer.in_sizes), xq_s) and torch.equal(_dense(w_mod, layer.in_sizes), w_mod_s)
    assert rel_fro(out, out_s) <= BF16_REL and rel_fro(gx, gx_s) <= BF16_REL
    assert rel_fro(grads["weight"], grads_s["weight"]) <= BF16_REL


@pytest.mark.parametrize("base,over", [
    ("bf16_static_adc", dict(in_shape=(130, 777), out_features=515, max_input_size=260, ir_init_value=2.0)),
    ("bf16_dynamic_eval", dict(in_shape=(65, 1001), out_features=70, max_input_size=512)),
    ("bf16_discretize", dict(in_shape=(200, 300), out_features=131, max_input_size=77, ir_init_value=2.0)),
    ("bf16_learnable_clip", dict(in_shape=(70, 500), out_features=33, max_input_size=250, ir_init_value=2.0)),
])
def test_ragged_layer_matches_oracle(base, over):
    from aihwkit_lightning_b200 import _lib
    from aihwkit_lightning_b200.nn import functional as F

    case = dict(C.CASES_BY_NAME[base], weight_scale=0.05, steps=1)
    case.update(over, noise_type="None", out_noise=0.0)  # replayed noise would keep the layer on the CUDA cores
    data = C.make_inputs(case)
    rec, grads = oracle_run(case, data)
    layer, x, out = run_product_layer(case, dict(data, w_noise=[None], out_noise=[None]))
    rows, k = x.shape
    desc = F.make_desc(layer.rpu_config, rows, k, data["n"], len(layer.in_sizes), torch.bfloat16, case["training"])
    assert _lib.load().al_operand_pitch(desc, _lib.tile_ends_array(layer.in_sizes)) > 0
    check_close("out", out, rec.out, torch.bfloat16, case)
    check_close("grad_x", x.grad, grads["grad_x"], torch.bfloat16, case)
    check_close("grad_w", layer.weight.grad, grads["grad_w"], torch.bfloat16, case)


def test_operand_pitch_is_checked_on_the_host():
    from aihwkit_lightning_b200 import _lib
    from aihwkit_lightning_b200.nn import functional as F

    lib = _lib.load()
    layer = _layer(1001, 515, 512, OPTIONS["train"])
    ends = _lib.tile_ends_array(layer.in_sizes)
    desc = F.make_desc(layer.rpu_config, 130, 1001, 515, 2, torch.bfloat16, False)
    assert lib.al_operand_pitch(desc, ends) == 2 * 504
    with F.operator_settings(engine="simt"):
        other = F.make_desc(layer.rpu_config, 130, 1001, 515, 2, torch.bfloat16, False)
    assert lib.al_operand_pitch(other, ends) == 0  # another engine: the dense layout
    # beyond 8192 rows a training call with few products a row stays with the CUDA cores, an evaluation does not
    for rows, k, n, train, pitch in ((8193, 1001, 515, True, 1008), (8192, 100, 10, True, 104), (8193, 100, 10, True, 0),
                                     (8193, 100, 100, True, 104), (8193, 100, 10, False, 104), (8193, 27, 16, False, 0),
                                     (8192, 27, 16, False, 32), (8193, 296, 1, True, 37 * 8), (8193, 296, 1, False, 37 * 8)):
        tiles = [8] * 37 if k == 296 else [k] if k < 1001 else layer.in_sizes
        tall = F.make_desc(layer.rpu_config, rows, k, n, len(tiles), torch.bfloat16, train)
        tall.save_for_backward = int(train)
        assert lib.al_operand_pitch(tall, _lib.tile_ends_array(tiles)) == pitch, (rows, k, n, train)
    even = F.make_desc(layer.rpu_config, 130, 1024, 512, 2, torch.bfloat16, False)
    ends = _lib.tile_ends_array([512, 512])
    even.engine = _lib.AL_ENGINE_PITCHED  # announced for a layer that has no pitched layout
    assert lib.al_operand_pitch(even, ends) == 0
    args = _lib.AlForwardArgs()
    buf = torch.zeros(4 << 20, device="cuda", dtype=torch.uint8)
    args.x = args.w = args.out = args.xq = args.w_mod = args.ir_rows = buf.data_ptr()
    args.tile_ends = ends
    assert lib.al_forward(even, args, None) != _lib.AL_OK


@pytest.mark.parametrize("rows,k,n,tile", [(65536, 1000, 1281, 250), (262144, 500, 100, -1), (1024, 1001, 20001, -1),
                                           (2048, 16385, 515, -1), (2048, 24601, 130, -1)],
                         ids=["rows_many_blocks", "rows_few_blocks", "channels", "features", "features_narrow"])
def test_long_sums_are_not_truncated(rows, k, n, tile):
    """Outputs and gradients are sums over features, rows or channels, in chunks of 8192 terms.  The tensor core adds 16
    terms at a time into a truncated accumulator: each of the 512 additions of a chunk shortens its sum by up to an ulp
    (2^-23; half of one on average, of a sum that grows like the root of the terms so far, so a third of 512 * 2^-23 =
    2e-5 of the whole); roundings of the bf16 result have no direction.  A sum in one accumulator loses four and more
    times as much."""
    layer = _layer(k, n, tile, OPTIONS["plain"])
    layer.train()
    layer.bias.data.zero_()
    gen = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(rows, k, device="cuda", generator=gen, dtype=torch.float32).bfloat16()
    g = torch.randn(rows, n, device="cuda", generator=gen, dtype=torch.float32).bfloat16()
    out, gx, grads, xq, w_mod = _pass(layer, x, g, "auto")
    assert xq.shape[1] != k  # on the tensor cores
    xq, w_mod = _dense(xq, layer.in_sizes), _dense(w_mod, layer.in_sizes).double()
    inside = x.abs() < 2.5  # the static range blocks the others
    exact_w = torch.zeros(n, k, device="cuda", dtype=torch.float64)
    shrink, size, square, count = [0.0, 0.0], [0.0, 0.0], [0.0, 0.0], [0, 0]

    def add(i, value, exact):
        shrink[i] += (exact.abs() - value.double() * exact.sign()).sum().item()
        size[i] += exact.abs().sum().item()
        square[i] += (value.double() - exact).square().sum().item()
        count[i] += exact.numel()

    for a in range(0, rows, 8192):
        rr = slice(a, a + 8192)
        exact_w += g[rr].double().t() @ xq[rr].double()
        if len(layer.in_sizes) == 1:  # more tiles: rounded to bf16 after each
            add(0, out[rr], xq[rr].double() @ w_mod.t())
        add(1, gx[rr][inside[rr]], (g[rr].double() @ w_mod)[inside[rr]])
    shrink.append(0.0), size.append(0.0), square.append(0.0), count.append(0)
    add(2, grads["weight"], exact_w)
    for i in range(3):
        if count[i]:
            noise = 4.0 * (square[i] ** 0.5) / size[i]  # four standard errors of a sum of independent roundings
            assert abs(shrink[i] / size[i]) <= 2e-5 + noise, (i, shrink[i] / size[i], noise)
