"""corr_index_forward of float64 volumes at the radii of its own kernel, at tiles of 64 pixels and
ragged ones, small and thin targets, against the float64 oracle (windows are blended in FP32: 1e-5
of the largest value).
"""

import numpy as np
import pytest
import torch

import oracle.corr as oc
from hislam2_b200 import backends

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h1,w1,h2,w2", [(1, 1, 1, 1, 1), (3, 8, 8, 5, 9), (2, 5, 13, 43, 2), (1, 16, 13, 16, 13), (2, 9, 7, 1, 70)])
@pytest.mark.parametrize("r", [3, 4])
def test_forward(cuda, n, h1, w1, h2, w2, r):
    g = torch.Generator().manual_seed(h1 + w2)
    vol = torch.randn(n, h1, w1, h2, w2, generator=g).double()
    coords = torch.stack([-4 + (w2 + 8) * torch.rand(n, h1, w1, generator=g), -4 + (h2 + 8) * torch.rand(n, h1, w1, generator=g)], 1)
    coords[0, :, 0, 0] = torch.tensor([1e9, -1e9]) if h1 * w1 > 1 else torch.tensor([0.5, 0.25])
    out, = backends.corr_index_forward(vol.to(cuda), coords.to(cuda), r)
    ref = oc.corr_index_forward(vol.numpy(), coords.numpy(), r)
    assert out.dtype == torch.float64 and np.abs(out.cpu().numpy() - ref).max() <= 1e-5 * np.abs(ref).max()
