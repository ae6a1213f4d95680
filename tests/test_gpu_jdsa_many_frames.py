"""JDSA on windows on both sides of the number of source frames from which its depth terms are summed
edge by edge ahead of the step: copies of a small window side by side, with and without source
frames missing at the ends, against the float64 oracle with the bars of the other JDSA tests; a bad
edge, and source frames missing in the middle, where the oracle's system is not positive definite, are
refused with the scales as they were.
"""

import pytest
import torch

from hislam2_b200 import mono, synth
from oracle import jdsa as ojdsa
from test_gpu_jdsa_cluster import args_of, rel

pytestmark = pytest.mark.gpu


def side_by_side(copies, grid, keep=None):
    p = synth.make_jdsa_problem("tiny6", hs=grid[0], ws=grid[1])
    K, out = p["poses"].shape[0], dict(p)
    for k in ("poses", "disps", "disps_prior", "dscales"):
        out[k] = p[k].repeat(copies, *[1] * (p[k].dim() - 1))
    shift = (K * torch.arange(copies))[:, None]
    at = [(p[k][None] + shift).reshape(-1) for k in ("ii", "jj")]
    live = torch.ones(len(at[0]), dtype=torch.bool) if keep is None else keep(at[0])
    out["ii"], out["jj"] = at[0][live], at[1][live]
    out["targets"], out["weights"] = (p[k].repeat(copies, 1, 1, 1)[live] for k in ("targets", "weights"))
    frames = torch.unique(out["ii"])
    out["eta"] = p["eta"].repeat(copies, 1, 1)[:len(frames)].contiguous()
    return out, len(frames)


@pytest.mark.parametrize("copies,grid,keep,frames", [(12, (2, 2), None, 72), (13, (2, 2), None, 78),
                                                     (13, (3, 4), lambda i: i > 2, 75),
                                                     (40, (2, 3), lambda i: i < 239, 239)])
def test_step_matches_oracle(cuda, copies, grid, keep, frames):
    p, M = side_by_side(copies, grid, keep)
    assert M == frames
    a = {k: (v.numpy().copy() if torch.is_tensor(v) else v) for k, v in p.items()}
    r = ojdsa.jdsa(a["targets"], a["weights"], a["eta"], a["poses"], a["disps"], a["intrinsics"], a["disps_prior"],
                   a["dscales"], a["ii"], a["jj"], a["alpha"])
    out, scales, cov = mono.JDSA(*args_of(p, cuda))
    assert rel(out.cpu(), r["disps"]) < 1e-5
    assert rel(scales.cpu().double() - torch.as_tensor(a["dscales"]).double(), r["dscales"] - a["dscales"]) < 1e-3
    assert rel(cov.cpu(), r["dzcov"]) < 1e-4


def test_gaps_are_refused_as_by_the_oracle(cuda):
    p, M = side_by_side(13, (2, 2), lambda i: i % 26 != 3)
    assert M == 75
    args = args_of(p, cuda)
    with pytest.raises(RuntimeError, match="positive definite"):
        mono.JDSA(*args)
    assert torch.equal(args[7].cpu(), p["dscales"])


def test_bad_edge_is_refused(cuda):
    p, _ = side_by_side(13, (2, 2))
    p["jj"][5] = 1000
    args = args_of(p, cuda)
    with pytest.raises(RuntimeError, match="outside"):
        mono.JDSA(*args)
    assert torch.equal(args[7].cpu(), p["dscales"])
