"""The lookups' outputs can be changed in place (a network applies an activation to them), with
the gradients of the operation out of place.  On the CPU with the kernels replaced by
plain torch, and with the kernels on the GPU.
"""

import pytest
import torch

from hislam2_b200 import backends
from hislam2_b200.corr import CorrBlock, CorrLookup
from test_corr_inplace_coords import plain_backward, plain_forward


def plain_volume(f1, f2, num_levels, precision):
    n, c, h, w = f1.shape
    vol = torch.einsum("nchw,ncyx->nhwyx", f1 / 4, f2 / 4)
    out = [vol]
    for _ in range(1, num_levels):
        v = out[-1]
        out.append(torch.nn.functional.avg_pool2d(v.reshape(n, h * w, *v.shape[3:]), 2, 2).reshape(n, h, w, v.shape[3] // 2,
                                                                                                v.shape[4] // 2))
    return out


def inputs(dev, dtype):
    g = torch.Generator().manual_seed(1)
    f1, f2 = ((torch.randn(1, 2, 128, 8, 9, generator=g) / 128 ** 0.5).to(dtype).to(dev) for _ in range(2))
    return f1, f2, (7 * torch.rand(1, 2, 8, 9, 2, generator=g)).to(dev)


def outputs(dev, dtype):
    f1, f2, coords = inputs(dev, dtype)
    f1.requires_grad_(True)
    yield f1, CorrLookup.apply(f1, f2, coords, 3, 2)
    block = CorrBlock(f1.detach(), f2, 2, 3)
    block.corr_pyramid = [v.requires_grad_(True) for v in block.corr_pyramid]
    yield block.corr_pyramid[0], block(coords)


def check(dev, dtype, differentiate):
    for (_, plain), (leaf, out) in zip(outputs(dev, dtype), outputs(dev, dtype)):
        assert not out._is_view()
        want = (0.5 * plain).relu()
        out *= 0.5
        out.relu_()
        assert torch.equal(out, want) and tuple(out.shape) == (1, 2, 2 * 49, 8, 9)
        if differentiate:
            assert torch.autograd.grad(out.float().sum(), leaf)[0].abs().max() > 0


def test_plain(monkeypatch):
    monkeypatch.setattr(backends, "corr_pyramid_fits", lambda *a: True)
    monkeypatch.setattr(backends, "corr_pyramid_forward", plain_forward)
    monkeypatch.setattr(backends, "corr_index_backward", plain_backward)
    monkeypatch.setattr(backends, "corr_volume", plain_volume)
    check(torch.device("cpu"), torch.float32, False)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["f16", "bf16"])
def test_kernels(cuda, dtype):
    check(cuda, dtype, True)
