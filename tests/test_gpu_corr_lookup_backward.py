"""CorrLookup's gradients in one pass over the levels (corr_lookup_backward) against float64
autograd through the pooled features, over tile edges, ragged grids whose pooled levels drop
a row or column, 1 to 4 levels, radii, types and non-contiguous inputs; and the per-level
route that other radii take.

Tolerance relative to the largest gradient: 1e-5 (FP32 sums of a few thousand terms) plus
half the spacing of the gradients' type.
"""

import pytest
import torch
import torch.nn.functional as F

from hislam2_b200 import backends
from hislam2_b200.corr import CorrLookup

pytestmark = pytest.mark.gpu


def reference(f1, f2, coords, grad, r, L):
    """Float64 gradients: bilinear windows of f1 . pooled f2 / 16, by grid gather."""
    a, b = (t.detach().double().requires_grad_(True) for t in (f1, f2))
    N, C, H, W = a.shape
    out, lv = [], b
    for i in range(L):
        if i:
            lv = F.avg_pool2d(lv, 2, stride=2)
        h, w = lv.shape[-2:]
        vol = torch.einsum("ncp,ncq->npq", a.flatten(2), lv.flatten(2)) / 16
        c = coords.double().reshape(N, H * W, 2) / 2 ** i
        x0, y0 = torch.floor(c[..., 0]), torch.floor(c[..., 1])
        fx, fy = (c[..., 0] - x0)[..., None, None], (c[..., 1] - y0)[..., None, None]
        k = torch.arange(-r, r + 2, device=a.device)
        x, y = (x0.long()[..., None] + k)[..., :, None], (y0.long()[..., None] + k)[..., None, :]
        ok = (x >= 0) & (x < w) & (y >= 0) & (y < h)
        at = (y.clamp(0, h - 1) * w + x.clamp(0, w - 1)).flatten(2)
        V = torch.gather(vol, 2, at).view(N, H * W, len(k), len(k)) * ok
        o = (1 - fx) * (1 - fy) * V[..., :-1, :-1] + (1 - fx) * fy * V[..., :-1, 1:] \
            + fx * (1 - fy) * V[..., 1:, :-1] + fx * fy * V[..., 1:, 1:]
        out.append(o.flatten(2).transpose(1, 2).reshape(N, -1, H, W))
    return torch.autograd.grad(torch.cat(out, 1), [a, b], grad.double())


def problem(N, H, W, r, L, dtype, dev, seed=0):
    g = torch.Generator().manual_seed(seed + H)
    f1, f2 = (torch.randn(N, 128, H, W, generator=g).to(dtype).to(dev) for _ in range(2))
    y, x = torch.meshgrid(torch.arange(H).float(), torch.arange(W).float(), indexing="ij")
    coords = (torch.stack([x, y], -1) + 2 * torch.randn(N, 1, 1, 2, generator=g) + torch.randn(N, H, W, 2, generator=g)).to(dev)
    coords[0, 0, 0] = -50.0
    grad = torch.randn(N, L * (2 * r + 1) ** 2, H, W, generator=g).to(dtype).to(dev)
    return f1, f2, coords, grad


@pytest.mark.parametrize("dtype,ulp", [(torch.float16, 2 ** -11), (torch.bfloat16, 2 ** -8), (torch.float32, 0.0)],
                         ids=["f16", "bf16", "f32"])
@pytest.mark.parametrize("N,H,W,r,L", [(2, 16, 16, 4, 4), (3, 9, 15, 3, 3), (1, 8, 9, 6, 4), (2, 1, 1, 2, 1), (1, 21, 11, 0, 2)])
def test_lookup_backward(cuda, N, H, W, r, L, dtype, ulp):
    f1, f2, coords, grad = problem(N, H, W, r, L, dtype, cuda)
    assert backends.corr_lookup_backward_fits(f1, r, L)
    got = backends.corr_lookup_backward(f1, f2, coords, grad, r, L)
    for a, b in zip(got, reference(f1, f2, coords, grad, r, L)):
        assert a.dtype == dtype
        assert (a.double() - b).abs().max() <= (1e-5 + ulp) * b.abs().max()


@pytest.mark.parametrize("r", [3, 7])
def test_corr_lookup_function_routes(cuda, r):
    """CorrLookup with permuted inputs, at a radius of each route."""
    f1, f2, coords, grad = problem(4, 10, 12, r, 2, torch.float16, cuda)
    a = f1.view(2, 2, 128, 10, 12).transpose(3, 4).contiguous().transpose(3, 4).requires_grad_(True)
    b = f2.view(2, 2, 128, 10, 12).requires_grad_(True)
    out = CorrLookup.apply(a, b, coords.view(2, 2, 10, 12, 2), r, 2)
    got = torch.autograd.grad(out, [a, b], grad.view(2, 2, -1, 10, 12))
    for x, y in zip(got, reference(f1, f2, coords, grad, r, 2)):
        assert (x.reshape(y.shape).double() - y).abs().max() <= (1e-5 + 2 ** -11) * y.abs().max()
