"""Weights, biases, gradients and replayed noise that start anywhere in an allocation (views into a flat buffer): the kernels
that read them in vectors give what they give for aligned copies."""
import pytest
import torch

from util import rel_fro

pytestmark = pytest.mark.gpu


def _off_by_one(t):
    flat = torch.empty(t.numel() + 1, device=t.device, dtype=t.dtype)
    view = flat[1:].view(t.shape)
    view.copy_(t)
    assert view.data_ptr() % 16
    return view


def _rpu(adc, static):
    from aihwkit_lightning_b200.simulator.configs import TorchInferenceRPUConfig

    rpu = TorchInferenceRPUConfig()
    rpu.mapping.max_input_size = 256
    rpu.forward.inp_res = 254.0
    if adc:
        rpu.forward.out_res, rpu.forward.out_bound = 254.0, 10.0
    irp = rpu.pre_post.input_range
    irp.enable, irp.dynamic = True, not static
    if static:
        irp.learn_input_range, irp.init_value, irp.init_from_data = True, 2.5, 0
    return rpu


@pytest.mark.parametrize("adc,static", [(False, False), (True, False), (False, True)])
def test_fp32_weights_bias_and_gradient(adc, static):
    from aihwkit_lightning_b200 import _lib
    from aihwkit_lightning_b200.nn import AnalogLinear
    from aihwkit_lightning_b200.nn import functional as F

    torch.manual_seed(0)
    layer = AnalogLinear(512, 520, bias=True, rpu_config=_rpu(adc, static), device="cuda", dtype=torch.float32).train()
    desc = F.make_desc(layer.rpu_config, 520, 512, 520, 2, torch.float32, True)
    assert _lib.load().al_uses_tcgen05(desc, _lib.tile_ends_array(layer.in_sizes))
    x, g = torch.randn(520, 512, device="cuda"), torch.randn(520, 520, device="cuda")
    results = []
    for make in (torch.clone, _off_by_one):
        layer.weight.data, layer.bias.data = make(layer.weight.data), make(layer.bias.data)
        layer.zero_grad(set_to_none=True)
        xs = make(x).requires_grad_(True)
        out = layer(xs)
        out.backward(make(g))
        results.append([out.detach(), xs.grad] + [p.grad for p in layer.parameters() if p.grad is not None])
    for i, (a, b) in enumerate(zip(*results)):
        if a.dim() == 1:  # column and range sums: vectors or single elements per thread, so another order of fp32 sums
            assert rel_fro(a, b) <= 1e-6
        else:
            assert torch.equal(a, b), i


@pytest.mark.parametrize("rows,adc", [(64, False), (300, True), (4096, True)])
def test_bf16_bias(rows, adc):
    from aihwkit_lightning_b200.nn import AnalogLinear

    torch.manual_seed(0)
    layer = AnalogLinear(512, 1032, bias=True, rpu_config=_rpu(adc, False), device="cuda", dtype=torch.bfloat16).eval()
    x = torch.randn(rows, 512, device="cuda").bfloat16()
    with torch.no_grad():
        want = layer(x)
        layer.bias.data = _off_by_one(layer.bias.data)
        assert torch.equal(layer(x), want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_replayed_output_noise(dtype):
    from aihwkit_lightning_b200.nn import AnalogLinear
    from aihwkit_lightning_b200.nn import functional as F

    rpu = _rpu(False, False)
    rpu.forward.out_noise = 0.1
    torch.manual_seed(0)
    layer = AnalogLinear(512, 520, bias=False, rpu_config=rpu, device="cuda", dtype=dtype).train()
    x = torch.randn(520, 512, device="cuda").to(dtype)
    noise = torch.randn(2, 520, 520, device="cuda").to(dtype)
    outs = []
    for z in (noise, _off_by_one(noise)):
        with torch.no_grad(), F.operator_settings(out_noise=z):
            outs.append(layer(x))
    assert torch.equal(*outs)
