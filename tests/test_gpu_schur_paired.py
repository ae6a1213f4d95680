"""The tensor-core Gram's two forms at the edges between them: frames of 20 to 43 Schur rows (one M
tile up to 21, two above, the SIMT Gram beyond 42), on grids that give a unit one pixel chunk,
several accumulators or a ragged last one, in one window.

The reduced camera matrix against the float64 oracle, before damping, 1e-6 of the largest entry
(3xTF32 products, FP32 sums over at most a few hundred pixels, combined in FP64).  The right-hand
side carries the linearisation's FP32 residuals, so the Gram's part of it is compared with the
SIMT Gram of the same rows: FP32 sums of up to 128 pixels there, 128 * 2^-24 < 1e-5 of the sum
of the terms' magnitudes.
"""

import numpy as np
import pytest
import torch

from hislam2_b200 import _lib, backends, synth
from oracle import ba as oba

pytestmark = pytest.mark.gpu


def star(K, ht, wd, seed):
    """K frames, every frame an edge from and to frame 0, and neighbours."""
    g = torch.Generator().manual_seed(seed)
    intr = synth.intrinsics_for((8 * ht, 8 * wd))
    gt = synth.se3_exp(0.03 * torch.randn(K, 6, generator=g, dtype=torch.float64))
    disps = 0.3 + torch.rand(K, ht, wd, generator=g, dtype=torch.float64)
    e = [(0, j) for j in range(1, K)] + [(j, 0) for j in range(1, K)] + [(j, j - 1) for j in range(2, K)]
    ii, jj = (torch.tensor([p[k] for p in e]) for k in (0, 1))
    xy = synth.reproject(gt, disps, intr, ii, jj)
    xy = xy + 0.5 * torch.randn(xy.shape, generator=g, dtype=torch.float64)
    f = lambda t: t.float().contiguous()  # noqa: E731
    return dict(poses=f(gt), disps=f(disps), intrinsics=f(intr), targets=f(xy.permute(0, 3, 1, 2)),
                weights=f(torch.rand(len(e), 2, ht, wd, generator=g)), eta=torch.full((K, ht, wd), 1e-3), ii=ii, jj=jj)


@pytest.mark.parametrize("K,ht,wd", [(3, 3, 5), (5, 43, 77), (10, 30, 40), (20, 9, 11), (21, 20, 33), (22, 20, 33),
                                     (23, 12, 16), (42, 8, 9), (43, 6, 7)])
def test_reduced_system(cuda, K, ht, wd):
    w = star(K, ht, wd, K)
    names = ("poses", "disps", "intrinsics", "targets", "weights", "eta")
    args = [w[k].to(cuda) for k in names] + [w["ii"].to(cuda), w["jj"].to(cuda), 0, K]
    A, b = backends.ba_reduced_system(*args)
    try:
        _lib.set_schur_path(1)
        _, simt_b = backends.ba_reduced_system(*args)
    finally:
        _lib.set_schur_path(0)
    r = oba.ba(*[w[k].double().numpy() for k in names], w["ii"].numpy(), w["jj"].numpy(), 0, K, 1, 1e-4, 0.1, trace=True)
    it = r.traces[0]
    assert np.abs(A.cpu().numpy() - (it["A"] - it["S"])).max() <= 1e-6 * np.abs(it["A"]).max()
    terms = np.einsum("ndp,np->nd", np.abs(it["E"]), np.abs(it["Q"] * it["w"])[r.kk_exp])
    assert float((b - simt_b).abs().max()) <= 1e-5 * terms.max()
