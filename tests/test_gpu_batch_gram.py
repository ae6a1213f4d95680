"""The batched solver's Schur Gram at the edges of its row counts: depth frames whose rows
(6 per edge or window pose, one for the right-hand side) sit on both sides of its stage
sizes (32 and 96 rows), of one tile per thread (176 rows) and of its limit (256 rows, the
general Gram above), on grids with ragged pixel counts; several windows per launch.

Against the float64 oracle, first iteration; tolerance 1e-4 relative to the largest
magnitude (the bar of the FP32 form).
"""

import math

import numpy as np
import pytest
import torch

import oracle
from hislam2_b200 import backends, synth

pytestmark = pytest.mark.gpu


def star(K, ht, wd, seed):
    """K frames, every frame an edge from and to frame 0."""
    g = torch.Generator().manual_seed(seed)
    intr = synth.intrinsics_for((8 * ht, 8 * wd))
    gt = synth.se3_exp(0.03 * torch.randn(K, 6, generator=g, dtype=torch.float64))
    disps = 0.3 + torch.rand(K, ht, wd, generator=g, dtype=torch.float64)
    ii = torch.tensor([0] * (K - 1) + list(range(1, K)))
    jj = torch.tensor(list(range(1, K)) + [0] * (K - 1))
    xy = synth.reproject(gt, disps, intr, ii, jj)
    xy = xy + 0.5 * torch.randn(xy.shape, generator=g, dtype=torch.float64)
    poses = synth.pose_compose(synth.se3_exp(0.01 * torch.randn(K, 6, generator=g, dtype=torch.float64)), gt)
    f = lambda t: t.float().contiguous()  # noqa: E731
    return dict(poses=f(poses), disps=f(disps), intrinsics=f(intr), targets=f(xy.permute(0, 3, 1, 2)),
                weights=f(torch.rand(len(ii), 2, ht, wd, generator=g)), eta=torch.full((K, ht, wd), 1e-3), ii=ii, jj=jj,
                t0=0, t1=K)


def rel(a, b):
    return float(np.abs(a.double().cpu().numpy() - b).max() / np.abs(b).max())


# rows of frame 0: 6 K + 1
@pytest.mark.parametrize("split", [1, 3])
def test_batch_gram_row_counts(cuda, split):
    sizes = [(2, 5, 9), (5, 7, 11), (6, 8, 16), (15, 7, 11), (16, 5, 13), (28, 6, 9), (30, 7, 7), (42, 5, 9), (43, 5, 7)]
    assert [6 * K + 1 for K, _, _ in sizes] == [13, 31, 37, 91, 97, 169, 181, 253, 259]
    cpu = [star(K, h, w, K) for K, h, w in sizes]
    ws = [{k: (v.to(cuda) if torch.is_tensor(v) else v) for k, v in w.items()} for w in cpu]
    plan = backends.BABatch(ws, 1e-4, 0.1, gram_split=split)
    plan.run(1)
    for w, (dx, dz), gpu in zip(cpu, plan.results(), ws):
        a = [w[k].double().numpy() for k in ("poses", "disps", "intrinsics", "targets", "weights", "eta")]
        r = oracle.ba.ba(*a, w["ii"].numpy(), w["jj"].numpy(), 0, w["t1"], 1, 1e-4, 0.1)
        assert math.isfinite(float(dz.abs().sum()))
        assert rel(dx, r.dx) < 1e-4 and rel(dz, r.dz) < 1e-4, w["t1"]
        assert rel(gpu["poses"], r.poses) < 1e-4 and rel(gpu["disps"], r.disps) < 1e-4, w["t1"]
