"""Infinities and NaN in the all-level lookup and the volume's epilogue: a tap that is not finite reaches
exactly the outputs whose four taps hold it (as by a blend of the same taps in torch), a feature
that is not finite exactly its pixels' rows of the volume and the pooled elements above them.
"""

import pytest
import torch
import torch.nn.functional as F

from hislam2_b200 import backends

pytestmark = pytest.mark.gpu


def taps(vol, planar, r):
    """(2r+2)^2 taps of vol [n, h1, w1, h2, w2] around floor(planar) - r, 0 outside: [n, y, x, h1, w1]."""
    n, h1, w1, h2, w2 = vol.shape
    k = torch.arange(2 * r + 2, device=vol.device)
    x = planar[:, 0].floor().long()[:, None, None] - r + k[None, None, :, None, None]
    y = planar[:, 1].floor().long()[:, None, None] - r + k[None, :, None, None, None]
    x, y = torch.broadcast_tensors(x, y)
    at = (y.clamp(0, h2 - 1) * w2 + x.clamp(0, w2 - 1)).permute(0, 3, 4, 1, 2).reshape(n, h1, w1, -1)
    v = torch.gather(vol.reshape(n, h1, w1, -1), 3, at).reshape(n, h1, w1, 2 * r + 2, 2 * r + 2).permute(0, 3, 4, 1, 2)
    return torch.where((x >= 0) & (x < w2) & (y >= 0) & (y < h2), v, torch.zeros_like(v))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16], ids=["f32", "f16", "bf16"])
@pytest.mark.parametrize("r", [3, 4])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
def test_lookup(cuda, r, dtype, value):
    n, h, w, L = 2, 9, 11, 3
    g = torch.Generator().manual_seed(r)
    vols = [torch.randn(n, h, w, h >> i, w >> i, generator=g).to(dtype).to(cuda) for i in range(L)]
    for v in vols:
        v[torch.rand(v.shape, generator=g).to(cuda) < 0.02] = value
    coords = torch.stack([-2 + (w + 4) * torch.rand(n, h, w, generator=g), -2 + (h + 4) * torch.rand(n, h, w, generator=g)],
                         -1).to(cuda)
    out = backends.corr_pyramid_forward(vols, coords, r).reshape(n, L, 2 * r + 1, 2 * r + 1, h, w)
    planar = coords.permute(0, 3, 1, 2)
    for i, v in enumerate(vols):
        bad = ~torch.isfinite(taps(v.float(), planar / 2 ** i, r))
        held = bad[:, :-1, :-1] | bad[:, 1:, :-1] | bad[:, :-1, 1:] | bad[:, 1:, 1:]      # [n, y, x, h, w]
        assert held.any() and torch.equal(~torch.isfinite(out[:, i]), held.transpose(1, 2))


@pytest.mark.parametrize("precision", ["native"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["f16", "bf16"])
def test_volume(cuda, dtype, precision):
    H, W = 17, 33
    g = torch.Generator().manual_seed(1)
    f1, f2 = (torch.randn(2, 128, H, W, generator=g).to(dtype).to(cuda) for _ in range(2))
    f1[0, 3, 4, 5] = float("inf")
    f2[1, 7, 10, 32] = float("nan")
    levels = backends.corr_volume(f1, f2, num_levels=4, precision=precision)
    for l, v in enumerate(levels):
        v = v.reshape(2, H, W, H >> l, W >> l)
        want = torch.zeros(v.shape, dtype=torch.bool, device=cuda)
        want[0, 4, 5] = True
        if (10 >> l) < (H >> l) and (32 >> l) < (W >> l):
            want[1, :, :, 10 >> l, 32 >> l] = True
        assert torch.equal(~torch.isfinite(v), want), l
        if l:
            up = levels[l - 1].reshape(2 * H * W, 1, H >> (l - 1), W >> (l - 1))
            assert torch.equal(F.avg_pool2d(up, 2, 2).reshape(v.shape).isfinite(), v.isfinite())
