"""The on-the-fly correlation's tensor-core tile kernel at the edges of its position chunks and boxes,
and its all-levels launch (AltCorrBlock without gradients)."""

import numpy as np
import pytest
import torch

import oracle.corr as oc
from hislam2_b200 import backends, corr as hcorr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return torch.device("cuda")


def np64(t):
    return t.detach().double().cpu().numpy()


def problem(H, W, frames, edges, spread, dtype, dev, seed, B=1):
    """Features of std 1/sqrt(C) and coordinates of the pixel grid plus noise of `spread` pixels, beyond
    the borders too."""
    g = torch.Generator().manual_seed(seed)
    f = (torch.randn(B, frames, 128, H, W, generator=g) / np.sqrt(128)).to(dev, dtype)
    v, u = torch.meshgrid(torch.arange(H, dtype=torch.float32), torch.arange(W, dtype=torch.float32), indexing="ij")
    crd = torch.stack([u, v], -1) + spread * torch.randn(B, edges, H, W, 2, generator=g) + 1.3
    ii = torch.randint(0, frames, (edges,), generator=g)
    jj = torch.randint(0, frames, (edges,), generator=g)
    return f, crd.to(dev), ii.to(dev), jj.to(dev)


# 1 x 1 target: one position; 8 x 8 and 9 x 7: 64 and 63; 13 x 5: 65 (one chunk and a position more);
# 33 x 31 scattered: box of 1023; 33 x 32: 1056, above the staged limit; 43 x 61 noise of 1 and 30 pixels
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["f16", "bf16"])
@pytest.mark.parametrize("H,W,spread,r,levels", [
    (1, 1, 0.5, 3, 1), (8, 8, 2.0, 3, 4), (7, 9, 2.0, 8, 2), (5, 13, 3.0, 0, 3), (31, 33, 30.0, 3, 2),
    (32, 33, 30.0, 3, 3), (43, 61, 1.0, 4, 4), (43, 61, 30.0, 3, 4)])
def test_altcorr_levels_vs_oracle(cuda, dtype, H, W, spread, r, levels):
    """Exact products and FP32 sums: only the rounding of the stored output differs from the float64
    oracle on the same 16-bit pyramid (2^-10 relative for float16, 2^-7 for bfloat16).  The same
    launch per level gives the same bits."""
    f, crd, ii, jj = problem(H, W, 3, 3, spread, dtype, cuda, seed=H * W + r)
    blk = hcorr.AltCorrBlock(f, num_levels=levels, radius=r)
    with torch.no_grad():
        out = blk(crd, ii, jj)
    assert backends.altcorr_levels_fits(blk.packed, crd, ii, jj, r)
    assert out.dtype == dtype and tuple(out.shape) == (1, 3, levels * (2 * r + 1) ** 2, H, W)
    planar = crd.permute(0, 1, 4, 2, 3).contiguous()
    tol = 2 ** -10 if dtype == torch.float16 else 2 ** -7
    for l in range(levels):
        part = out[:, :, l * (2 * r + 1) ** 2:(l + 1) * (2 * r + 1) ** 2]
        one, = backends.altcorr_forward_packed(blk.packed[0], blk.packed[l], planar / 2 ** l, ii, jj, r)
        assert torch.equal(one.flatten(2, 3), part)
        ref = oc.altcorr_forward(np64(f), np64(blk.pyramid[l]), np64(planar / 2 ** l), ii.cpu().numpy(),
                                 jj.cpu().numpy(), r)
        ref = ref.reshape(np64(part).shape)
        assert np.abs(np64(part) - ref).max() <= tol * max(np.abs(ref).max(), 1e-30)


def test_altcorr_levels_batch_bad_index_strides(cuda):
    """Two batches, strided coordinates, an edge out of range (zeros), no edges."""
    f, crd, ii, jj = problem(11, 18, 4, 5, 1.0, torch.float16, cuda, seed=9, B=2)
    jj[3] = 4
    blk = hcorr.AltCorrBlock(f, num_levels=3, radius=3)
    strided = crd.permute(0, 1, 3, 2, 4).contiguous().permute(0, 1, 3, 2, 4)
    with torch.no_grad():
        out, again, none = blk(crd, ii, jj), blk(strided, ii, jj), blk(crd[:, :0], ii[:0], jj[:0])
    assert torch.equal(out, again) and none.shape == (2, 0, 147, 11, 18)
    assert torch.count_nonzero(out[:, 3]) == 0
    for b in range(2):
        alone = hcorr.AltCorrBlock(f[b:b + 1].contiguous(), num_levels=3, radius=3)
        with torch.no_grad():
            assert torch.equal(alone(crd[b:b + 1], ii, jj)[0], out[b])
