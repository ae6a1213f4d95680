"""The all-level lookup (corr_pyramid_forward, PyramidSampler) against the float64 oracle and
against one corr_index_forward per level, on volumes at both element parities (odd plane
sizes, views that start at an odd element), coordinates inside, across and far outside the
target, tiles of 64 pixels that end mid-way.

Tolerance relative to the largest value: 1e-5 in FP32, half the spacing of the type on top
for 16-bit outputs (2^-11, 2^-8): the taps are read exactly and blended in FP32.
"""

import numpy as np
import pytest
import torch

import oracle.corr as oc
from hislam2_b200 import backends
from hislam2_b200.corr import CorrBlock, CorrSampler

pytestmark = pytest.mark.gpu
TYPES = [(torch.float32, 1e-5), (torch.float16, 1e-5 + 2 ** -11), (torch.bfloat16, 1e-5 + 2 ** -8)]


def np64(t):
    return t.detach().double().cpu().numpy()


def levels(n, h, w, L, dtype, dev, seed, offset=0):
    g = torch.Generator().manual_seed(seed)
    out = []
    for i in range(L):
        shape = (n, h, w, h >> i, w >> i)
        flat = torch.randn(int(np.prod(shape)) + offset, generator=g).to(dtype).to(dev)
        out.append(flat[offset:].view(shape))           # offset 1: data pointer at an odd element
    return out


def coordinates(n, h, w, seed, dev):
    g = torch.Generator().manual_seed(seed + 1)
    c = torch.stack([-6 + (w + 12) * torch.rand(n, h, w, generator=g), -6 + (h + 12) * torch.rand(n, h, w, generator=g)], -1)
    c[0, 0, 0] = torch.tensor([1e9, -1e9])
    c[0, 0, 1 % w] = torch.tensor([2.0, 1.0])           # whole numbers
    c[0, -1, -1] = torch.tensor([w + 2.5, float(h)])
    return c.to(dev)


@pytest.mark.parametrize("dtype,tol", TYPES, ids=["f32", "f16", "bf16"])
@pytest.mark.parametrize("n,h,w,L,offset", [(2, 9, 11, 3, 0), (3, 8, 8, 4, 1), (1, 16, 13, 4, 1), (2, 5, 7, 2, 0), (1, 1, 2, 1, 1)])
@pytest.mark.parametrize("r", [3, 4])
def test_pyramid_lookup(cuda, n, h, w, L, offset, r, dtype, tol):
    vols = levels(n, h, w, L, dtype, cuda, r + h, offset)
    crd = coordinates(n, h, w, h, cuda)
    assert backends.corr_pyramid_fits(vols, crd, r)
    got = backends.corr_pyramid_forward(vols, crd, r)
    ref = oc.corr_block_lookup([np64(v) for v in vols], np64(crd)[None], r)[0]
    assert got.dtype == dtype and got.shape == ref.shape
    assert np.abs(np64(got) - ref).max() <= tol * np.abs(ref).max()
    planar = crd.permute(0, 3, 1, 2).contiguous()
    one = torch.cat([backends.corr_index_forward(v, planar / 2 ** i, r)[0].flatten(1, 2) for i, v in enumerate(vols)], 1)
    assert torch.equal(got, one)


@pytest.mark.parametrize("r,dtype", [(3, torch.float32), (2, torch.float32), (4, torch.float64), (4, torch.float16)])
def test_corr_block_call_takes_every_form(cuda, r, dtype):
    """Radii and types the all-level kernel does not take, permuted coordinates, and gradients."""
    h, w, L = 9, 10, 3
    block = CorrBlock.__new__(CorrBlock)
    block.num_levels, block.radius = L, r
    block.corr_pyramid = [v.requires_grad_(i != 1) for i, v in enumerate(levels(2, h, w, L, dtype, cuda, 3))]
    crd = coordinates(2, h, w, 5, cuda)[None]
    out = block(crd.permute(0, 1, 4, 2, 3).contiguous().permute(0, 1, 3, 4, 2))
    assert torch.equal(out, block(crd))
    planar = crd[0].permute(0, 3, 1, 2).contiguous()
    ref = torch.cat([CorrSampler.apply(v, planar / 2 ** i, r).view(1, 2, -1, h, w)
                     for i, v in enumerate(block.corr_pyramid)], 2)
    assert torch.equal(out, ref)
    g = torch.randn(out.shape, device=cuda).to(dtype)
    need = [v for v in block.corr_pyramid if v.requires_grad]
    for a, b in zip(torch.autograd.grad(out, need, g), torch.autograd.grad(ref, need, g)):
        assert torch.equal(a, b)
