"""The tiled gradients of the on-the-fly correlation (128 channels) against the float64
oracle, at the edges of the 8x8 tiles, for coordinates that follow the pixel grid (one
union of windows per 2x2 group) and scattered ones (separate windows).

Tolerances, relative to the largest gradient: 1e-5 in FP32 (a sum of at most a few
thousand terms of similar size, each rounded at 2^-24); half the spacing of the output
type on top for 16-bit gradients (2^-11, 2^-8).
"""

import numpy as np
import pytest
import torch

import droid_backends
import oracle.corr as oc

pytestmark = pytest.mark.gpu


def problem(B, N1, N2, H, W, H2, W2, M, seed, dev, dtype, spread):
    g = torch.Generator().manual_seed(seed)
    f1 = torch.randn(B, N1, 128, H, W, generator=g).to(dtype)
    f2 = torch.randn(B, N2, 128, H2, W2, generator=g).to(dtype)
    ii = torch.randint(0, N1, (M,), generator=g)
    jj = torch.randint(0, N2, (M,), generator=g)
    if spread is None:       # anywhere, partly outside
        crd = torch.stack([-3 + (W2 + 6) * torch.rand(B, M, H, W, generator=g),
                           -3 + (H2 + 6) * torch.rand(B, M, H, W, generator=g)], 2)
    else:                    # the pixel grid scaled to the target, moved by a few pixels
        y, x = torch.meshgrid(torch.arange(H).float() * H2 / H, torch.arange(W).float() * W2 / W, indexing="ij")
        crd = torch.stack([x, y]) + 4 * torch.randn(B, M, 2, 1, 1, generator=g) \
            + spread * torch.randn(B, M, 2, H, W, generator=g)
    return f1.to(dev), f2.to(dev), crd.to(dev).contiguous(), ii.to(dev), jj.to(dev)


def np64(t):
    return t.detach().double().cpu().numpy()


def close(a, ref, tol):
    return float(np.abs(np64(a) - ref).max()) <= tol * float(np.abs(ref).max())


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.float16, 1e-5 + 2 ** -11),
                                       (torch.bfloat16, 1e-5 + 2 ** -8)], ids=["f32", "f16", "bf16"])
@pytest.mark.parametrize("H,W,H2,W2,r,spread", [(8, 8, 8, 8, 3, 0.5), (7, 9, 3, 4, 4, 0.5), (17, 16, 17, 16, 4, 1.0),
                                                (9, 7, 9, 7, 6, None), (1, 1, 1, 1, 0, 0.1), (10, 23, 5, 11, 1, 2.0)])
def test_tiled_backward_vs_oracle(cuda, H, W, H2, W2, r, spread, dtype, tol):
    f1, f2, crd, ii, jj = problem(2, 3, 2, H, W, H2, W2, 4, r + H, cuda, dtype, spread)
    g = torch.randn(2, 4, 2 * r + 1, 2 * r + 1, H, W, generator=torch.Generator().manual_seed(5)).to(cuda)
    g1, g2 = droid_backends.altcorr_backward(f1, f2, crd, ii, jj, g, r, 1.0 / 16)
    assert g1.dtype == dtype and g1.shape == f1.shape and g2.shape == f2.shape
    r1, r2 = oc.altcorr_backward(np64(f1), np64(f2), np64(crd), ii.cpu().numpy(), jj.cpu().numpy(), np64(g), r,
                                 scale=1.0 / 16)
    assert close(g1, r1, tol) and close(g2, r2, tol)


def test_tiled_backward_unused_frames_and_bad_index(cuda):
    f1, f2, crd, ii, jj = problem(1, 5, 5, 9, 10, 9, 10, 2, 3, cuda, torch.float32, 0.5)
    ii[:], jj[:] = 1, 3
    ii[1] = 9                # outside the frames: contributes nothing
    g = torch.randn(1, 2, 7, 7, 9, 10, device=cuda)
    g1, g2 = droid_backends.altcorr_backward(f1, f2, crd, ii, jj, g, 3)
    r1, r2 = oc.altcorr_backward(np64(f1), np64(f2), np64(crd[:, :1]), [1], [3], np64(g[:, :1]), 3)
    assert close(g1, r1, 1e-5) and close(g2, r2, 1e-5)
    assert torch.count_nonzero(g1[:, [0, 2, 3, 4]]) == 0 and torch.count_nonzero(g2[:, [0, 1, 2, 4]]) == 0


def test_tiled_backward_keeps_infinities_in_their_windows(cuda):
    """An infinite feature reaches only the pixels whose window holds it (0 * inf elsewhere would be NaN)."""
    H, W, r = 16, 24, 2
    f1, f2, crd, ii, jj = problem(1, 1, 1, H, W, H, W, 1, 8, cuda, torch.float32, 0.2)
    f2[0, 0, 5, 4, 6] = float("inf")
    f1[0, 0, 7, 9, 11] = float("inf")
    g = torch.rand(1, 1, 2 * r + 1, 2 * r + 1, H, W, device=cuda) + 0.5
    g1, g2 = droid_backends.altcorr_backward(f1, f2, crd, ii, jj, g, r)
    x0, y0 = torch.floor(crd[0, 0, 0]) - r, torch.floor(crd[0, 0, 1]) - r
    holds = (x0 <= 6) & (6 < x0 + 2 * r + 2) & (y0 <= 4) & (4 < y0 + 2 * r + 2)
    assert torch.equal(~torch.isfinite(g1[0, 0, 5]), holds)
    assert torch.isfinite(g1[0, 0, [c for c in range(128) if c != 5]]).all()
    ys, xs = torch.meshgrid(torch.arange(H, device=cuda), torch.arange(W, device=cuda), indexing="ij")
    reach = (xs >= x0[9, 11]) & (xs < x0[9, 11] + 2 * r + 2) & (ys >= y0[9, 11]) & (ys < y0[9, 11] + 2 * r + 2)
    assert torch.equal(~torch.isfinite(g2[0, 0, 7]), reach)
