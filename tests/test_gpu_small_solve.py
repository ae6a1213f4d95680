"""The one-CTA solve of small reduced systems at the edges of its 16x16 blocks and of its range
(up to 224 unknowns; larger systems take the many-CTA solve), through ba (6 unknowns per pose)
and pgba (7, padded to an even count), and its rule for systems that are not positive definite.

Against the float64 oracle, one step; tolerance 1e-4 relative to the largest magnitude (the
FP32 assembly; the solve itself is FP64).
"""

import numpy as np
import pytest
import torch

import droid_backends
import oracle
from hislam2_b200 import synth
from oracle import pgba as opgba

pytestmark = pytest.mark.gpu
HT, WD = 6, 9


def window(K, seed):
    """K frames, edges to neighbours at distance 1, 2 and 5 both ways."""
    g = torch.Generator().manual_seed(seed)
    intr = synth.intrinsics_for((8 * HT, 8 * WD))
    gt = synth.se3_exp(0.03 * torch.randn(K, 6, generator=g, dtype=torch.float64))
    disps = 0.3 + torch.rand(K, HT, WD, generator=g, dtype=torch.float64)
    e = [(i, j) for i in range(K) for d in (1, 2, 5) for j in (i - d, i + d) if 0 <= j < K]
    ii, jj = (torch.tensor([p[k] for p in e]) for k in (0, 1))
    xy = synth.reproject(gt, disps, intr, ii, jj)
    xy = xy + 0.5 * torch.randn(xy.shape, generator=g, dtype=torch.float64)
    poses = synth.pose_compose(synth.se3_exp(0.01 * torch.randn(K, 6, generator=g, dtype=torch.float64)), gt)
    f = lambda t: t.float().contiguous()  # noqa: E731
    return dict(poses=f(poses), disps=f(disps), intrinsics=f(intr), targets=f(xy.permute(0, 3, 1, 2)),
                weights=f(torch.rand(len(e), 2, HT, WD, generator=g)), eta=torch.full((K, HT, WD), 1e-3), ii=ii, jj=jj)


def rel(a, b):
    return float(np.abs(a.double().cpu().numpy() - b).max() / max(np.abs(b).max(), 1e-30))


NAMES = ("poses", "disps", "intrinsics", "targets", "weights", "eta")


@pytest.mark.parametrize("P", [1, 2, 3, 8, 16, 21, 24, 37, 38])
def test_ba_small_systems(cuda, P):
    w = window(P + 1, P)
    d = {k: v.to(cuda) for k, v in w.items()}
    dx, dz, _ = droid_backends.ba(*[d[k] for k in NAMES], d["ii"], d["jj"], 1, P + 1, 1, 1e-4, 0.1, False)
    r = oracle.ba.ba(*[w[k].double().numpy() for k in NAMES], w["ii"].numpy(), w["jj"].numpy(), 1, P + 1, 1, 1e-4, 0.1)
    assert rel(dx, r.dx) < 1e-4 and rel(dz, r.dz) < 1e-4
    assert rel(d["poses"], r.poses) < 1e-4 and rel(d["disps"], r.disps) < 1e-4


@pytest.mark.parametrize("P", [1, 5, 31, 32])
def test_pgba_small_systems(cuda, P):
    w = window(P + 1, 50 + P)
    g = torch.Generator().manual_seed(P)
    w["poses"] = torch.cat([w["poses"], torch.exp(0.05 * torch.randn(P + 1, 1, generator=g))], 1).contiguous()
    iip, jjp = torch.arange(0, P), torch.arange(1, P + 1)
    J = torch.randn(2, P, 7, 7, generator=g, dtype=torch.float64)
    wJ = J.transpose(2, 3)
    res = 0.01 * torch.randn(P, 7, 1, generator=g, dtype=torch.float64)
    Hsp = torch.stack([wJ[0] @ J[0], wJ[0] @ J[1], wJ[1] @ J[0], wJ[1] @ J[1]])[:, None].float().contiguous()
    vsp = -torch.stack([wJ[0] @ res, wJ[1] @ res]).squeeze(-1)[:, None].float().contiguous()
    d = {k: v.to(cuda) for k, v in w.items()}
    dx, dz = droid_backends.pgba(*[d[k] for k in NAMES], Hsp.to(cuda), vsp.to(cuda), d["ii"], d["jj"], iip.to(cuda),
                                 jjp.to(cuda), 1, P + 1, 1e-4, 0.1)
    r = opgba.pgba(*[w[k].double().numpy() for k in NAMES], Hsp.numpy(), vsp.numpy(), w["ii"].numpy(), w["jj"].numpy(),
                   iip.numpy(), jjp.numpy(), 1, P + 1, 1e-4, 0.1)
    assert rel(dx, r.dx) < 1e-4 and rel(dz, r.dz) < 1e-4


@pytest.mark.parametrize("P", [2, 20, 37])
def test_not_positive_definite_gives_no_update(cuda, P):
    """lm = -2 makes every damped diagonal negative: poses stay, dx = 0, whichever block fails first."""
    w = window(P + 1, 90)
    d = {k: v.to(cuda) for k, v in w.items()}
    dx, _, _ = droid_backends.ba(*[d[k] for k in NAMES], d["ii"], d["jj"], 1, P + 1, 1, -2.0, 0.0, True)
    assert torch.count_nonzero(dx) == 0
    assert (d["poses"].cpu() - w["poses"]).abs().max() <= 1e-6
