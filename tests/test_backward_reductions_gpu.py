"""Reductions of the backward pass against float64 sums: the bias gradient (column sums over a cluster of CTAs) and
the gradient of a static input range with its straight-through zeroing."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("m,n", [(1, 1), (7, 63), (129, 64), (512, 1024), (1000, 1500), (1023, 65), (4097, 260)])
def test_bias_gradient_is_the_column_sum(dtype, m, n):
    from aihwkit_lightning_b200 import _lib

    lib = _lib.load()
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    g = torch.randn(m, n, device="cuda", generator=gen).to(dtype)
    out = torch.full((n + 8,), 7.0, device="cuda", dtype=dtype)
    desc = _lib.AlDesc()
    desc.M, desc.K, desc.N, desc.T = m, 8, n, 1
    desc.dtype = _lib.AL_F32 if dtype == torch.float32 else _lib.AL_BF16
    desc.inp_res = desc.out_res = desc.out_bound = -1.0
    args = _lib.AlBackwardArgs()
    args.tile_ends = _lib.tile_ends_array([8])
    args.grad_out, args.grad_bias = g.data_ptr(), out.data_ptr()
    _lib.check(lib.al_backward(desc, args, torch.cuda.current_stream().cuda_stream))
    want, scale = g.double().sum(0), g.double().abs().sum(0)
    # a chain of at most m / 32 additions per thread, 64 row groups and 8 CTAs, each rounding to 2^-24 of the partial
    # sum (below the sum of magnitudes); bf16 results round once more
    bound = (m / 32 + 80) * 2.0 ** -24 * scale + (2.0 ** -8 * want.abs() if dtype == torch.bfloat16 else 0)
    assert bool(((out[:n].double() - want).abs() <= bound).all())
    assert bool((out[n:] == 7.0).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("m,k,tiles", [(1, 8, 1), (31, 72, 3), (33, 75, 2), (2500, 1024, 8)])
def test_static_range_gradient_and_clipped_inputs(dtype, m, k, tiles):
    from aihwkit_lightning_b200.nn import AnalogLinear
    from aihwkit_lightning_b200.simulator.configs import TorchInferenceRPUConfig

    rpu = TorchInferenceRPUConfig()
    rpu.mapping.max_input_size = -(-k // tiles)
    irp = rpu.pre_post.input_range
    irp.enable, irp.dynamic, irp.learn_input_range, irp.init_value, irp.init_from_data = True, False, True, 1.5, 0
    irp.decay = 0.0
    torch.manual_seed(k)
    layer = AnalogLinear(k, 16, bias=False, rpu_config=rpu).to(device="cuda", dtype=dtype).train()
    x = torch.randn(m, k, device="cuda").to(dtype).requires_grad_(True)
    g = torch.randn(m, 16, device="cuda").to(dtype)
    layer(x).backward(g)
    full = torch.empty(m, k, device="cuda", dtype=dtype)  # the gradient before the clipped entries were zeroed
    full.copy_(g.float() @ layer.weight.float())
    xd, clipped = x.detach().double(), x.detach().abs() >= 1.5
    assert bool((x.grad[clipped & (x.detach().abs() != 1.5)] == 0).all())
    assert bool((x.grad[~clipped] != 0).float().mean() > 0.9)
    lo = 0
    tol = 1e-5 if dtype == torch.float32 else 2e-2  # fp32 sums of products; bf16 gradients and results
    for t, size in enumerate(layer.in_sizes):
        cols = slice(lo, lo + size)
        gx, xt = full[:, cols].double(), xd[:, cols]
        want = 1.5 * (gx[xt >= 1.5].clamp(max=0).sum() - gx[xt <= -1.5].clamp(min=0).sum())
        scale = 1.5 * gx[clipped[:, cols]].abs().sum() + 1e-6
        assert abs(layer.input_range.grad[t].double() - want) <= tol * scale
        lo += size


@pytest.mark.parametrize("m,rows", [(3, (0, 1, 2)), (18976, (0, 8, 16)), (18976, (0, 1, 18975)), (9, (0, 1, 8))],
                         ids=["row_per_warp", "rows_of_a_warp", "two_blocks", "two_short_blocks"])
def test_range_gradient_keeps_small_terms_between_large_ones(m, rows):
    """Rows of 2^24, 1 and -2^24: fp32 sums over rows lose the 1, which the result consists of."""
    _range_gradient(m, rows, (2.0 ** 24, 1.0, -(2.0 ** 24)), 1.0)


@pytest.mark.parametrize("values,want", [((math.inf, 1.0, -2.0), math.inf), ((1.0, -math.inf, 2.0), -math.inf),
                                         ((3e38, 3e38, 3e38), math.inf)])
def test_range_gradient_of_infinite_gradients(values, want):
    _range_gradient(18976, (0, 1, 18975), values, want)


def _range_gradient(m, rows, values, want):
    from aihwkit_lightning_b200 import _lib

    lib = _lib.load()
    k = 32
    x = torch.zeros(m, k, device="cuda")
    g = torch.zeros(m, 1, device="cuda")
    for row, v in zip(rows, values):
        x[row, 5], g[row, 0] = 2.0, v
    w, ir = torch.ones(1, k, device="cuda"), torch.ones(1, device="cuda")
    grad_x, grad_ir = torch.empty(m, k, device="cuda"), torch.empty(1, device="cuda")
    scratch = torch.empty(lib.al_backward_scratch_floats(m, k, 1, 1), device="cuda")
    desc = _lib.AlDesc()
    desc.M, desc.K, desc.N, desc.T = m, k, 1, 1
    desc.dtype, desc.ir_mode, desc.engine = _lib.AL_F32, _lib.AL_IR_FAST, _lib.AL_ENGINE_SIMT
    desc.inp_res, desc.out_res, desc.out_bound = 254.0, -1.0, -1.0
    args = _lib.AlBackwardArgs()
    args.tile_ends = _lib.tile_ends_array([k])
    args.grad_out, args.x, args.w_mod, args.ir_rows = g.data_ptr(), x.data_ptr(), w.data_ptr(), ir.data_ptr()
    args.grad_x, args.grad_input_range = grad_x.data_ptr(), grad_ir.data_ptr()
    args.reduce_scratch, args.reduce_scratch_floats = scratch.data_ptr(), scratch.numel()
    _lib.check(lib.al_backward(desc, args, torch.cuda.current_stream().cuda_stream))
    assert grad_ir.item() == want
    assert not bool(grad_x[x > 1].any())


@pytest.mark.parametrize("m,n", [(262144, 16), (262144, 10), (262144, 65), (65537, 33), (16385, 64), (8191, 130), (255, 3)])
def test_bias_gradient_of_tall_matrices(m, n):
    """Against float64, to the error of a sum whose chain of roundings is one per 256 rows, then 256 partial sums (with and
    without a workspace, which decides how the rows are split).  A rounding is uniform in half an ulp of the partial
    sum at hand: its rms is 2^-24 / sqrt(3) of that sum at most, and the sum grows like the root of the rows in it, so
    c roundings on the way to s leave at most 2^-24 / sqrt(3) * s * sqrt(c / 2) (rms over the columns)."""
    from aihwkit_lightning_b200 import _lib

    lib = _lib.load()
    desc = _lib.AlDesc()
    desc.M, desc.K, desc.N, desc.T = m, 8, n, 1
    desc.dtype, desc.inp_res, desc.out_res, desc.out_bound = _lib.AL_F32, -1.0, -1.0, -1.0
    args = _lib.AlBackwardArgs()
    args.tile_ends = _lib.tile_ends_array([8])
    scratch = torch.empty(lib.al_backward_scratch_floats(m, 8, n, 1), device="cuda")
    for workspace in (False, True):
        if workspace:
            args.reduce_scratch, args.reduce_scratch_floats = scratch.data_ptr(), scratch.numel()
        square, values = 0.0, 0
        for seed in range(max(1, 256 // n)):  # a few hundred sums: the rms is known to some 5 %
            gen = torch.Generator(device="cuda").manual_seed(seed)
            g = torch.randn(m, n, device="cuda", generator=gen)
            out = torch.empty(n, device="cuda")
            args.grad_out, args.grad_bias = g.data_ptr(), out.data_ptr()
            _lib.check(lib.al_backward(desc, args, torch.cuda.current_stream().cuda_stream))
            square += ((out.double() - g.double().sum(0)) ** 2).sum().item()
            values += n
        chain = min(m, 256) + (m + 255) // 256
        assert (square / values) ** 0.5 <= 2.0 ** -24 / 3 ** 0.5 * m ** 0.5 * (chain / 2) ** 0.5
