"""The extension behind ``nn.functional``: arguments it refuses before anything is launched (no GPU needed)."""
import ctypes

import pytest
import torch


def test_arguments_are_checked():
    from aihwkit_lightning_b200 import _lib

    host = _lib.host()
    for fn, count in ((host.forward, 26), (host.backward, 18)):
        with pytest.raises(ValueError):
            fn()
        with pytest.raises(TypeError):  # no descriptor
            fn(*[None] * count)
        with pytest.raises(ValueError):  # a descriptor that is too small
            fn((ctypes.c_int32 * 1)(), (ctypes.c_int32 * 1)(), *[None] * (count - 2))
        desc, ends = _lib.AlDesc(), (ctypes.c_int32 * 1)(8)
        desc.M, desc.K, desc.N, desc.T = 4, 8, 8, 2
        with pytest.raises(ValueError):  # two tiles announced, one end given
            fn(desc, ends, *[None] * (count - 2))
        desc.T = 1
        with pytest.raises(TypeError):  # weights / gradient missing
            fn(desc, ends, *[None] * (count - 2))
        with pytest.raises(TypeError):  # not a tensor
            fn(desc, ends, 1.5, 1.5, *[None] * (count - 4))


def test_layer_refuses_cpu_tensors():
    from aihwkit_lightning_b200.nn import AnalogLinear
    from aihwkit_lightning_b200.simulator.configs import TorchInferenceRPUConfig

    with pytest.raises(ValueError):
        AnalogLinear(8, 8, rpu_config=TorchInferenceRPUConfig())(torch.zeros(2, 8))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(3, 1024, 16), (3, 16, 1024), (2, 65, 33), (2, 33, 65), (1, 1, 1), (5, 64, 64), (2, 130, 3), (1, 7, 2049)])
def test_transpose_images(shape, dtype):
    from aihwkit_lightning_b200.nn import functional as F

    src = torch.randn(*shape, device="cuda").to(dtype)
    assert torch.equal(F._transpose_images(src, *shape), src.transpose(-1, -2).contiguous())


@pytest.mark.gpu
def test_static_ranges_are_copied_back_only_where_they_were_copied():
    """The library updates a contiguous range in place; a strided one goes through a copy and back."""
    from torch.utils._python_dispatch import TorchDispatchMode

    from aihwkit_lightning_b200.nn import AnalogLinear
    from aihwkit_lightning_b200.simulator.configs import TorchInferenceRPUConfig

    class Copies(TorchDispatchMode):
        count = 0

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.count += func is torch.ops.aten.copy_.default
            return func(*args, **(kwargs or {}))

    rpu = TorchInferenceRPUConfig()
    rpu.mapping.max_input_size, rpu.forward.inp_res = 16, 254.0
    irp = rpu.pre_post.input_range
    irp.enable, irp.learn_input_range, irp.init_value, irp.init_from_data = True, True, 3.0, 10
    ranges = []
    for strided in (False, True):
        torch.manual_seed(0)
        layer = AnalogLinear(64, 32, bias=False, rpu_config=rpu, device="cuda", dtype=torch.float32).train()
        if strided:
            layer.input_range.data = torch.full((8,), 3.0, device="cuda")[::2]
            assert not layer.input_range.is_contiguous()
        with Copies() as copies, torch.no_grad():
            layer(torch.randn(40, 64, device="cuda"))
        assert (copies.count > 0) == strided
        ranges.append(layer.input_range.detach().clone())
    assert torch.equal(*ranges) and not bool((ranges[0] == 3.0).any())  # updated from the data


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_convolution_takes_gradients_of_any_layout(dtype):
    """The operator transposes the gradient of its images: one that is not contiguous gives what its copy gives."""
    from aihwkit_lightning_b200.nn import AnalogConv2d
    from aihwkit_lightning_b200.simulator.configs import TorchInferenceRPUConfig

    rpu = TorchInferenceRPUConfig()
    rpu.mapping.max_input_size, rpu.forward.inp_res = 64, 254.0
    rpu.pre_post.input_range.enable = rpu.pre_post.input_range.dynamic = True
    torch.manual_seed(0)
    conv = AnalogConv2d(8, 20, 3, padding=1, rpu_config=rpu, device="cuda", dtype=dtype).train()
    x = torch.randn(3, 8, 9, 7, device="cuda").to(dtype)
    g = torch.randn(3, 20, 9, 7, device="cuda").to(dtype)
    layouts = [g, g.contiguous(memory_format=torch.channels_last), g.transpose(2, 3).contiguous().transpose(2, 3),
               torch.cat([g, g], dim=1)[:, 20:], g[:, :, :1, :1].expand(3, 20, 9, 7)]
    for grad in layouts:
        results = []
        for gg in (grad, grad.clone(memory_format=torch.contiguous_format)):
            conv.zero_grad()
            xs = x.clone().requires_grad_(True)
            conv(xs).backward(gg)
            results.append((xs.grad, conv.weight.grad.clone(), conv.bias.grad.clone()))
        for a, b in zip(*results):
            assert torch.equal(a, b)
