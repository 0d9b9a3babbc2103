"""fp32 layers on the tensor cores: DAC codes as exact bf16 integers, weights and upstream gradients as
bf16 planes, fp32 accumulation -- against the CPU oracle to the fp32 bar (1e-5 relative), with the
noise replayed.  Static and dynamic input ranges, ADC clamp masks folded into the gradient planes, bias,
per-channel scales, multi-dimensional inputs, row counts and widths that are not multiples of the block
sizes; benchmark configuration 1 at its own size; forward and backward kernels on single CTAs (blocks of 32, 64 and 128
columns) and on CTA pairs."""
import re

import pytest
import torch

import cases as C
from test_parity_gpu import check_close
from util import oracle_run, rel_fro, run_product_layer

pytestmark = pytest.mark.gpu

CASES = [
    ("static_train_noise", dict(in_shape=(512, 1024), out_features=1024, max_input_size=512, ir_init_value=3.0,
                                weight_scale=1 / 32)),                       # configuration 1
    ("static_train_noise_pc", dict(in_shape=(512, 1024), out_features=1024, max_input_size=512, ir_init_value=3.0,
                                   weight_scale=1 / 32, out_noise_per_channel=False)),
    ("static_train_noise_pc", dict(in_shape=(192, 640), out_features=320, max_input_size=160, ir_init_value=2.0)),
    ("dynamic_adc_noise", dict(in_shape=(256, 1024), out_features=512, max_input_size=256)),
    ("dynamic_adc_gauss_pc_clip", dict(in_shape=(200, 512), out_features=264, max_input_size=128)),
    ("static_adc", dict(in_shape=(130, 512), out_features=520, max_input_size=128, ir_init_value=2.0)),
    ("dynamic_3d_input", dict(in_shape=(3, 50, 256), out_features=136, max_input_size=64)),
    ("dynamic_plain_eval", dict(in_shape=(300, 384), out_features=200, max_input_size=128)),
    ("static_init_from_data", dict(in_shape=(256, 512), out_features=256, max_input_size=256)),
    ("no_bias", dict(in_shape=(128, 256), out_features=128, max_input_size=-1)),
    # single CTAs: 64 columns (128 blocks of them, twice as many of 32), then 128 columns (several rounds of either)
    ("static_train_noise", dict(in_shape=(1000, 256), out_features=1016, max_input_size=128, ir_init_value=2.0)),
    ("dynamic_adc_noise", dict(in_shape=(2000, 256), out_features=2040, max_input_size=128)),
]


@pytest.mark.parametrize("base,over", CASES, ids=[f"{b}-{'x'.join(map(str, o['in_shape']))}x{o['out_features']}" for b, o in CASES])
@pytest.mark.parametrize("engine", ["tcgen05_single", "tcgen05_pair"])
def test_fp32_layer_on_tensor_cores_matches_oracle(base, over, engine):
    case = dict(C.CASES_BY_NAME[base])
    case.setdefault("weight_scale", 0.05)
    case["weight_scale"] = 0.05
    case.update(over)
    case["steps"] = 1
    data = C.make_inputs(case)
    rec, grads = oracle_run(case, data, w_noise=data["w_noise"][-1], out_noise=data["out_noise"][-1])
    capture = {}
    layer, x, out = run_product_layer(case, data, engine=engine, capture=capture)
    assert capture["uses_tcgen05"]
    dtype = data["dtype"]
    assert dtype == torch.float32
    check_close("out", out, rec.out, dtype, case)
    check_close("grad_x", x.grad, grads["grad_x"], dtype, case)
    check_close("grad_w", layer.weight.grad, grads["grad_w"], dtype, case)
    if case["bias"]:
        check_close("grad_bias", layer.bias.grad, grads["grad_bias"], dtype, case)
    if grads["grad_ir"] is not None and case["ir_learn"]:
        assert torch.allclose(layer.input_range.grad.cpu(), grads["grad_ir"], rtol=1e-4, atol=1e-5)


def test_auto_engine_picks_the_tensor_cores_for_a_large_fp32_layer_and_agrees_with_the_cuda_cores():
    from aihwkit_lightning_b200.nn import AnalogLinear
    from aihwkit_lightning_b200.nn import functional as F
    from util import NS

    case = dict(C.DEFAULTS)
    case.update(ir_dynamic=True, inp_res=254.0, max_input_size=512, out_bound=10.0, out_res=254.0)
    rpu = C.build_rpu_config(NS, case)
    torch.manual_seed(0)
    layer = AnalogLinear(1024, 768, bias=True, rpu_config=rpu).cuda().eval()
    x = torch.randn(640, 1024, device="cuda", requires_grad=True)
    g = torch.randn(640, 768, device="cuda")
    results = {}
    for engine in ("auto", "simt"):
        cap = {}
        layer.zero_grad(set_to_none=True)
        x.grad = None
        with F.operator_settings(engine=engine, capture=cap):
            out = layer(x)
        out.backward(g)
        results[engine] = (cap["uses_tcgen05"], out.detach(), x.grad.clone(), layer.weight.grad.clone())
    assert results["auto"][0] and not results["simt"][0]
    # ADC on: a last-ulp difference of an accumulator may move an output by one converter level
    flips = (results["auto"][1] != results["simt"][1]).float().mean().item()
    assert flips < 5e-3 or rel_fro(results["auto"][1], results["simt"][1]) < 1e-5
    assert rel_fro(results["auto"][2], results["simt"][2]) < 2e-3
    assert rel_fro(results["auto"][3], results["simt"][3]) < 2e-3


def _layer(k, n, tile, out_noise=0.0, per_channel_clip=False, bias=True):
    from aihwkit_lightning_b200.nn import AnalogLinear
    from aihwkit_lightning_b200.simulator.configs import TorchInferenceRPUConfig
    from aihwkit_lightning_b200.simulator.enums import WeightClipType

    rpu = TorchInferenceRPUConfig()
    rpu.mapping.max_input_size = tile
    rpu.forward.inp_res, rpu.forward.out_noise = 254.0, out_noise
    rpu.pre_post.input_range.enable = rpu.pre_post.input_range.dynamic = True
    if per_channel_clip:
        rpu.clip.type, rpu.clip.sigma = WeightClipType.LAYER_GAUSSIAN_PER_CHANNEL, 100.0
    torch.manual_seed(7)
    return AnalogLinear(k, n, bias=bias, rpu_config=rpu, device="cuda", dtype=torch.float32)


@pytest.mark.parametrize("rows,n,columns", [(512, 1024, 32), (1024, 1024, 64), (2048, 2048, 128)])
def test_engines_run_the_forward_kernel_they_name(rows, n, columns):
    from aihwkit_lightning_b200.nn import functional as F

    layer, x = _layer(256, n, 128).eval(), torch.randn(rows, 256, device="cuda")
    outs, ran = {}, {}
    for engine in ("tcgen05_single", "tcgen05_pair"):
        with torch.no_grad(), F.operator_settings(engine=engine):
            layer(x)
            with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
                outs[engine] = layer(x)
                torch.cuda.synchronize()
        names = " ".join(e.key for e in prof.key_averages())
        # rounding type, output stage, pairs, element type, ragged, columns staged per CTA
        ran[engine] = re.search(r"fwd_tc_kernel<\d+, -?\d+, (\w+), \d+, \w+, (\d+)[,>]", names).groups()
    assert ran == {"tcgen05_single": ("false", str(columns)), "tcgen05_pair": ("true", "64")}
    # one order of the sum over k on either
    assert rel_fro(outs["tcgen05_single"], outs["tcgen05_pair"]) <= 1e-6


SIZES = [(1000, 256, 1016, 128), (2050, 1024, 1096, 256), (520, 512, 264, 512)]


@pytest.mark.parametrize("engine", ["tcgen05_single", "tcgen05_pair"])
@pytest.mark.parametrize("shape", SIZES, ids=lambda s: "x".join(map(str, s)))
def test_output_noise_of_the_compiled_output_stage(shape, engine):
    """Without ADC and clamp the output stage is fixed at compile time and draws its noise from the library's generator:
    the same values as the stage that reads every switch at run time (which a per-channel clip type selects, without
    effect on a layer that has no bound); one standard normal per output and tile, independent of its neighbours."""
    from aihwkit_lightning_b200.nn import functional as F

    rows, k, n, tile = shape
    x = torch.randn(rows, k, device="cuda")
    outs = {}
    with torch.no_grad(), F.operator_settings(engine=engine):
        for name, per_channel in (("compiled", False), ("run_time", True)):
            layer = _layer(k, n, tile, out_noise=0.1, per_channel_clip=per_channel).train()
            torch.cuda.manual_seed(5)
            outs[name] = layer(x)
            outs[name + "_next"] = layer(x)
        clean = layer.eval()(x)
    assert rel_fro(outs["compiled"], outs["run_time"]) <= 1e-6
    assert rel_fro(outs["compiled_next"], outs["run_time_next"]) <= 1e-6
    w, sizes = layer.weight.detach(), layer.in_sizes
    var, lo = torch.zeros(rows, device="cuda"), 0
    for size in sizes:  # s_t = out_noise / sqrt(T) * range of the row * largest weight of the tile
        cols = slice(lo, lo + size)
        var += (w[:, cols].abs().max() * 0.1 / len(sizes) ** 0.5 * x[:, cols].abs().amax(1)) ** 2
        lo += size
    z, z2 = ((outs[key] - clean) / var.sqrt()[:, None] for key in ("compiled", "compiled_next"))
    z, z2 = z.double(), z2.double()
    # five standard errors of each statistic of rows * n independent standard normals
    five = 5.0 / (rows * n) ** 0.5
    assert abs(z.mean().item()) <= five
    assert abs(z.var().item() - 1.0) <= five * 2 ** 0.5 + 1e-4
    assert abs((z ** 4).mean().item() - 3.0) <= five * 96 ** 0.5 + 1e-3
    for a, b in ((z, z2), (z[1:], z[:-1]), (z[:, 1:], z[:, :-1]), (z[:, 8:], z[:, :-8]), (z[128:], z[:-128])):
        assert abs((a * b).mean().item()) <= 1.2 * five  # fewer products than outputs
    # every row and every column on its own: the largest of a few thousand variances
    for dim, count in ((0, rows), (1, n)):
        v = z.var(dim=dim)
        assert bool(((v - 1.0).abs() <= 6.0 * (2.0 / count) ** 0.5).all())
