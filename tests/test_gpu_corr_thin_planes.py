"""corr_index_forward on thin targets, whose longer side passes 2^20: windows at both ends, across
the middle and out of the target, at either element parity, against windows cut from the volume in
float64.  Tolerance: 1e-5 of the largest value in FP32 (exact taps, an FP32 blend), half
the type's spacing on top in FP16.
"""

import pytest
import torch

from hislam2_b200 import backends

pytestmark = pytest.mark.gpu


def windows(vol, x, y, r):
    """Bilinear (2r+1)^2 windows (x slowest) of vol [h2, w2] around one point, float64."""
    h, w = vol.shape
    x0, y0 = int(x // 1), int(y // 1)
    fx, fy = x - x0, y - y0
    v = torch.zeros(2 * r + 2, 2 * r + 2, dtype=torch.float64)
    for a in range(2 * r + 2):
        for b in range(2 * r + 2):
            if 0 <= x0 - r + a < w and 0 <= y0 - r + b < h:
                v[a, b] = vol[y0 - r + b, x0 - r + a].double().cpu()
    return ((1 - fx) * (1 - fy) * v[:-1, :-1] + (1 - fx) * fy * v[:-1, 1:] + fx * (1 - fy) * v[1:, :-1]
            + fx * fy * v[1:, 1:])


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.float16, 1e-5 + 2 ** -11)], ids=["f32", "f16"])
@pytest.mark.parametrize("h2,w2", [(1, (1 << 20) + 101), (3, 1 << 21), ((1 << 20) + 101, 1), (1 << 21, 4)])
@pytest.mark.parametrize("r", [3, 4])
def test_thin_target(cuda, h2, w2, r, dtype, tol):
    h1, w1 = 1, 7
    g = torch.Generator().manual_seed(h2 % 1000 + r)
    vol = torch.randn(1, h1, w1, h2, w2, generator=g).to(dtype).to(cuda)
    long = max(h2, w2)
    at = torch.tensor([0.25, long - 1.5, long / 2 + 0.5, (1 << 20) + 40.5, -r - 0.5, long + r - 0.25, 3.0 * long])
    across = torch.tensor([0.5, 0.0, 0.25, 0.75, 0.0, -0.5, 0.0])
    x, y = (at, across) if w2 >= h2 else (across, at)
    coords = torch.stack([x, y]).view(1, 2, h1, w1).to(cuda)
    out, = backends.corr_index_forward(vol, coords, r)
    ref = torch.stack([windows(vol[0, 0, p], float(x[p]), float(y[p]), r) for p in range(w1)], -1)
    assert ref.abs().max() > 0 and ref[..., -1].abs().max() == 0
    assert (out[0, :, :, 0].double().cpu() - ref).abs().max() <= tol * ref.abs().max()
