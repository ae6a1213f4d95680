"""The clustered JDSA step at the edges of its splits: edge lists longer than a scan and a batch,
frames smaller and larger than one round of the cluster, several cells, windows with frames
that have no edges; and the keys it makes on the device, wrong counts included."""

import numpy as np
import pytest
import torch

from hislam2_b200 import mono, synth
from oracle import jdsa as ojdsa

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.abs(np.asarray(a, np.float64) - b).max() / max(np.abs(b).max(), 1e-30))


def args_of(p, cuda):
    d = {k: v.to(cuda) if torch.is_tensor(v) else v for k, v in p.items()}
    return [d[k] for k in ("targets", "weights", "eta", "poses", "disps", "intrinsics", "disps_prior", "dscales", "ii",
                           "jj", "alpha")]


# (window, copies of its edges, scale grid, source frames kept): tiny6 has 192 pixels a frame, so one CTA of
# the cluster has pixels and 16 copies are 58 edges a frame and more; frontend has 3311, two rounds
CASES = [("tiny6", 1, (2, 2), None), ("tiny6", 16, (3, 3), None), ("tiny6", 32, (2, 8), None),
         ("frontend_small", 12, (4, 4), None), ("frontend", 3, (3, 2), None),
         ("frontend_small", 2, (2, 2), lambda i: i < 3)]


@pytest.mark.parametrize("name,copies,grid,keep", CASES)
def test_step_matches_oracle(cuda, name, copies, grid, keep):
    p = synth.make_jdsa_problem(name, hs=grid[0], ws=grid[1], keep=keep)
    for k in ("ii", "jj"):
        p[k] = p[k].repeat(copies)
    p["targets"] = p["targets"].repeat(copies, 1, 1, 1)
    p["weights"] = p["weights"].repeat(copies, 1, 1, 1) / copies
    a = {k: (v.numpy().copy() if torch.is_tensor(v) else v) for k, v in p.items()}
    r = ojdsa.jdsa(a["targets"], a["weights"], a["eta"], a["poses"], a["disps"], a["intrinsics"], a["disps_prior"],
                   a["dscales"], a["ii"], a["jj"], a["alpha"])
    out, scales, cov = mono.JDSA(*args_of(p, cuda))
    assert rel(out.cpu(), r["disps"]) < 1e-5
    assert rel(scales.cpu().double() - torch.as_tensor(a["dscales"]).double(), r["dscales"] - a["dscales"]) < 1e-3
    assert rel(cov.cpu(), r["dzcov"]) < 1e-4


def test_two_runs_are_equal(cuda):
    p = synth.make_jdsa_problem("frontend", hs=3, ws=3)
    a, b = (mono.JDSA(*args_of(dict(p, dscales=p["dscales"].clone()), cuda)) for _ in range(2))
    assert all(torch.equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("rows", [-1, 1])
def test_eta_of_another_count_is_refused(cuda, rows):
    p = synth.make_jdsa_problem("tiny6")
    M = len(torch.unique(p["ii"]))
    p["eta"] = torch.full((M + rows, *p["eta"].shape[1:]), 1e-3)
    args = args_of(p, cuda)
    with pytest.raises(RuntimeError, match="M = %d distinct" % M):
        mono.JDSA(*args)
    assert torch.equal(args[7].cpu(), p["dscales"])


@pytest.mark.parametrize("frame", [-1, 6, 1 << 40])
def test_source_frame_out_of_range_is_refused(cuda, frame):
    p = synth.make_jdsa_problem("tiny6")
    p["ii"] = torch.where(p["ii"] == p["ii"].max(), frame, p["ii"])
    args = args_of(p, cuda)
    with pytest.raises(RuntimeError, match="outside"):
        mono.JDSA(*args)
    assert torch.equal(args[7].cpu(), p["dscales"])
