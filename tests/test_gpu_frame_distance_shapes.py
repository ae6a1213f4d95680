"""frame_distance over its launch shapes (one, four and eight warps per edge), grids narrower than a
warp and ragged ones, self pairs, and points behind the camera, against the float64 oracle.
Tolerance 1e-5 relative, 1e-5 px absolute (FP32 image coordinates of up to 100 px, averaged)."""

import numpy as np
import pytest
import torch

import droid_backends
from hislam2_b200 import synth
from oracle import frame_distance as ofd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E", [1, 7, 8 * 148, 16 * 148 + 1, 32 * 148 + 3])
@pytest.mark.parametrize("ht,wd", [(43, 77), (3, 5), (1, 1), (9, 33)])
def test_frame_distance_shapes(cuda, E, ht, wd):
    g = torch.Generator().manual_seed(E + ht)
    K = 6
    poses = synth.se3_exp(0.1 * torch.randn(K, 6, generator=g, dtype=torch.float64)).float()
    poses[4, 2] = -3.0                                      # most of its points fall behind the camera
    disps = (0.1 + 1.5 * torch.rand(K, ht, wd, generator=g)).contiguous()
    intr = synth.intrinsics_for((8 * ht, 8 * wd)).float()
    pairs = torch.randint(0, K * K, (E,), generator=g)
    ii, jj = pairs // K, pairs % K
    d = droid_backends.frame_distance(poses.to(cuda), disps.to(cuda), intr.to(cuda), ii.to(cuda), jj.to(cuda), 0.3)
    kinds = torch.arange(K * K)
    ref = ofd.frame_distance(poses.double().numpy(), disps.double().numpy(), intr.double().numpy(),
                             (kinds // K).numpy(), (kinds % K).numpy(), 0.3)[pairs.numpy()]
    got = d.cpu().double().numpy()
    assert np.array_equal(got >= 1000, ref >= 1000)
    near = ref < 1000
    np.testing.assert_allclose(got[near], ref[near], rtol=1e-5, atol=1e-5)
