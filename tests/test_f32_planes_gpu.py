"""fp32 layers on the tensor cores: the passes that write codes and weight planes only, and the forward on CTA pairs,
against the CUDA-core kernels of the same layer (same weight noise, no output noise: the engines draw that differently)."""
import pytest
import torch

from util import rel_fro

pytestmark = pytest.mark.gpu

# two planes carry 16 significant bits of an operand: 2.2e-6 rms per product term, the bar of fp32 layers here is 1e-5
F32_REL = 1e-5

SHAPES = [
    (256, 2064, 512, 1032),   # tiles wider than a warp keeps in registers
    (512, 1040, 264, 520),    # a last group of lanes without work
    (1024, 4096, 40, 4096),   # fewer than 64 channels: the fp32 weights are written too
    (2050, 1024, 1096, 256),  # CTA pairs, ragged last blocks
]


@pytest.mark.parametrize("dynamic,bound", [(False, False), (True, True)], ids=["static", "dynamic_bound"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_matches_cuda_cores(shape, dynamic, bound):
    from aihwkit_lightning_b200.nn import AnalogLinear
    from aihwkit_lightning_b200.nn import functional as F
    from aihwkit_lightning_b200.simulator.configs import TorchInferenceRPUConfig
    from aihwkit_lightning_b200.simulator.enums import WeightNoiseInjectionType

    rows, k, n, tile = shape
    rpu = TorchInferenceRPUConfig()
    rpu.mapping.max_input_size = tile
    rpu.forward.inp_res = 254.0
    if bound:
        # the per-tile gradient planes of a layer with a clamp; a bound nothing reaches, because an output within 1e-5 of
        # it may be clamped by one order of the sum and not by the other, and one of the rows x n mask bits moves a
        # gradient by 1 / sqrt(rows n) = 3e-3
        rpu.forward.out_bound = 1e3
    irp = rpu.pre_post.input_range
    irp.enable, irp.dynamic = True, dynamic
    if not dynamic:
        irp.learn_input_range, irp.init_value, irp.init_from_data = True, 2.5, 0
    rpu.modifier.noise_type, rpu.modifier.std_dev = WeightNoiseInjectionType.ADD_NORMAL_PER_CHANNEL, 0.02
    torch.manual_seed(1)
    layer = AnalogLinear(k, n, bias=True, rpu_config=rpu, device="cuda", dtype=torch.float32).train()
    x0, g = torch.randn(rows, k, device="cuda"), torch.randn(rows, n, device="cuda")
    results = []
    for engine in ("auto", "simt"):
        layer.zero_grad()
        x = x0.clone().requires_grad_(True)
        torch.cuda.manual_seed(9)
        with F.operator_settings(engine=engine):
            out = layer(x)
            out.backward(g)
        results.append([out.detach(), x.grad] + [p.grad for p in layer.parameters() if p.grad is not None])
    for i, (a, b) in enumerate(zip(*results)):
        assert rel_fro(a, b) <= F32_REL, (i, rel_fro(a, b))
