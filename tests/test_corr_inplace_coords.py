"""CorrBlock's differentiable lookup keeps the coordinates it was called with: a caller that moves
its coordinates in place between the lookup and the backward (an update loop does) gets the
gradients at the old ones, whichever of the levels and coordinates need a gradient.  On the
CPU with the two kernels replaced by plain torch, and with the kernels on the GPU.
"""

import pytest
import torch
import torch.nn.functional as F

from hislam2_b200 import backends
from hislam2_b200.corr import CorrBlock


def sample(volume, planar, r):
    """corr_index_forward in plain torch: [N, 2r+1 (x), 2r+1 (y), H, W]."""
    n, h, w, h2, w2 = volume.shape
    d = torch.arange(-r, r + 1, dtype=torch.float32, device=volume.device)
    x = planar[:, 0].reshape(-1, 1, 1) + d[:, None]
    y = planar[:, 1].reshape(-1, 1, 1) + d[None]
    at = torch.stack([2 * (x + 0.5 * torch.ones_like(y)) / w2 - 1, 2 * (y + 0.5 * torch.ones_like(x)) / h2 - 1], -1)
    out = F.grid_sample(volume.reshape(-1, 1, h2, w2), at, align_corners=False)
    return out.reshape(n, h, w, 2 * r + 1, 2 * r + 1).permute(0, 3, 4, 1, 2).contiguous()


def plain_forward(volumes, coords, radius):
    h, w = coords.shape[-3:-1]
    planar = coords.reshape(-1, h, w, 2).permute(0, 3, 1, 2)
    out = torch.cat([sample(v, planar / 2 ** i, radius).flatten(1, 2) for i, v in enumerate(volumes)], 1)
    return torch.empty(*coords.shape[:-3], *out.shape[1:], dtype=out.dtype).copy_(out.reshape(*coords.shape[:-3], *out.shape[1:]))


def plain_backward(volume, planar, grad, radius):
    v = volume.detach().requires_grad_(True)
    with torch.enable_grad():
        return list(torch.autograd.grad(sample(v, planar, radius), [v], grad))


def check(dev, need_volumes, need_coords):
    n, h, w, r = 2, 6, 7, 3
    g = torch.Generator().manual_seed(0)
    block = CorrBlock.__new__(CorrBlock)
    block.num_levels, block.radius = 2, r
    block.corr_pyramid = [torch.randn(n, h, w, h >> i, w >> i, generator=g).to(dev).requires_grad_(i in need_volumes)
                          for i in range(2)]
    at = (6 * torch.rand(1, n, h, w, 2, generator=g)).to(dev)
    weight = torch.randn(1, n, 2 * (2 * r + 1) ** 2, h, w, generator=g).to(dev)
    need = [block.corr_pyramid[i] for i in need_volumes]
    grads = []
    for move in (False, True):
        coords = (at.clone().requires_grad_(True) if need_coords else at.clone()) * 1.0
        out = block(coords)
        if move:
            coords += 2.5
        grads.append(torch.autograd.grad(out, need, weight) if need else out.sum().backward() or ())
    for a, b in zip(*grads):
        assert a.abs().max() > 0 and torch.equal(a, b)


FORMS = [((0, 1), False), ((0,), False), ((1,), True), ((), True)]


@pytest.mark.parametrize("need_volumes,need_coords", FORMS)
def test_plain(monkeypatch, need_volumes, need_coords):
    monkeypatch.setattr(backends, "corr_pyramid_fits", lambda *a: True)
    monkeypatch.setattr(backends, "corr_pyramid_forward", plain_forward)
    monkeypatch.setattr(backends, "corr_index_backward", plain_backward)
    check(torch.device("cpu"), need_volumes, need_coords)


@pytest.mark.gpu
@pytest.mark.parametrize("need_volumes,need_coords", FORMS)
def test_kernels(cuda, need_volumes, need_coords):
    check(cuda, need_volumes, need_coords)
