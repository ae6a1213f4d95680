"""The 16-bit lookup at the two ends of a volume, whose words reach out of it when it starts or ends in
the middle of one: volumes of an odd and an even number of elements at both parities, with
infinities as their neighbours in memory, and windows that hold the first and the last element.  The
result is that of a volume of its own bit for bit, and finite.
"""

import pytest
import torch

from hislam2_b200 import backends

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["f16", "bf16"])
@pytest.mark.parametrize("n,h1,w1,h2,w2", [(1, 1, 1, 1, 1), (1, 1, 1, 1, 2), (1, 3, 3, 3, 5), (3, 5, 13, 7, 9), (2, 8, 8, 4, 6)])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("r", [3, 4])
def test_ends(cuda, n, h1, w1, h2, w2, offset, r, dtype):
    g = torch.Generator().manual_seed(n * h1 + w2)
    vol = torch.randn(n, h1, w1, h2, w2, generator=g).to(dtype).to(cuda)
    buf = torch.full((vol.numel() + 16,), float("inf"), dtype=dtype, device=cuda)
    placed = buf[8 + offset:8 + offset + vol.numel()].view(vol.shape)
    placed.copy_(vol)
    coords = torch.stack([w2 * torch.rand(n, h1, w1, generator=g), h2 * torch.rand(n, h1, w1, generator=g)], 1)
    coords[0, :, 0, 0] = torch.tensor([0.25, 0.5])
    coords[-1, :, -1, -1] = torch.tensor([w2 - 1.25, h2 - 1.5])
    coords = coords.to(cuda)
    out, = backends.corr_index_forward(placed, coords, r)
    want, = backends.corr_index_forward(vol, coords, r)
    assert torch.isfinite(out).all() and torch.equal(out, want)
    assert out[0, :, :, 0, 0].abs().max() > 0 and out[-1, :, :, -1, -1].abs().max() > 0
    whole, = backends.corr_index_forward(vol.float(), coords, r)
    assert (out.float() - whole).abs().max() <= (1e-5 + 2.0 ** (-11 if dtype == torch.float16 else -8)) * whole.abs().max()
