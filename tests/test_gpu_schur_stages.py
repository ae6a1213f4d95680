"""The tensor-core Gram of frames of two M tiles (more than 21 SE3 rows, 18 Sim3 rows), whose two splitting
groups take turns on three stages: many solves of one window in a row, on a grid of many pixel chunks
with the E rows partly out of the cache, all equal to the SIMT Gram's to 1e-4 of the largest increment
(the bar of the FP32 forms), none of them ending a wait early or late.
"""

import pytest
import torch

import droid_backends
from hislam2_b200 import _lib, synth

pytestmark = pytest.mark.gpu


def window(K, per_frame, ht, wd, seed, dev):
    g = torch.Generator().manual_seed(seed)
    intr = synth.intrinsics_for((8 * ht, 8 * wd))
    poses = synth.se3_exp(0.03 * torch.randn(K, 6, generator=g, dtype=torch.float64))
    disps = 0.3 + torch.rand(K, ht, wd, generator=g, dtype=torch.float64)
    ii = torch.arange(K).repeat_interleave(per_frame)
    jj = (ii + 1 + torch.arange(per_frame).repeat(K)) % K
    xy = synth.reproject(poses, disps, intr, ii, jj)
    xy = xy + 0.5 * torch.randn(xy.shape, generator=g, dtype=torch.float64)
    f = lambda t: t.float().contiguous().to(dev)  # noqa: E731
    return dict(poses=f(poses), disps=f(disps), intrinsics=f(intr), targets=f(xy.permute(0, 3, 1, 2)),
                weights=f(torch.rand(len(ii), 2, ht, wd, generator=g)), eta=torch.full((K, ht, wd), 1e-3, device=dev),
                ii=ii.to(dev), jj=jj.to(dev))


NAMES = ("poses", "disps", "intrinsics", "targets", "weights", "eta")


@pytest.mark.parametrize("K,per_frame,ht,wd,solves", [(120, 24, 43, 77, 60), (60, 35, 24, 32, 60), (40, 22, 60, 80, 60)])
def test_many_solves(cuda, K, per_frame, ht, wd, solves):
    w = window(K, per_frame, ht, wd, K, cuda)
    spoil = torch.empty(1 << 26, dtype=torch.uint8, device=cuda)

    def solve():
        poses, disps = w["poses"].clone(), w["disps"].clone()
        dx, dz = droid_backends.ba(poses, disps, *[w[k] for k in NAMES[2:]], w["ii"], w["jj"], 1, K, 1, 1e-4, 0.1, False)[:2]
        return dx.clone(), dz.clone()

    try:
        _lib.set_schur_path(1)
        want = solve()
    finally:
        _lib.set_schur_path(0)
    for k in range(solves):
        spoil.fill_(k & 127)
        for a, b in zip(solve(), want):
            assert float((a - b).abs().max()) <= 1e-4 * float(b.abs().max()), k
