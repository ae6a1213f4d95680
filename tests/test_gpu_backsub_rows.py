"""The back-substitution at the edges of its row lists (64 rows of a depth frame at a time, read two by
two) and of its pixel vectors (54 and 117 pixels: neither fills a vector), in ba and BABatch.

Frame 0 is tied to n frames in both directions.  One step against the float64 oracle; tolerance 1e-4
relative to the largest magnitude, as for the other FP32-assembled steps.
"""

import pytest
import torch

import droid_backends
import oracle
import test_gpu_small_solve as small
from hislam2_b200 import backends

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ht,wd", [(6, 9), (9, 13)])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 131])
def test_rows(cuda, monkeypatch, n, ht, wd):
    monkeypatch.setattr(small, "HT", ht)
    monkeypatch.setattr(small, "WD", wd)
    w = small.window(n + 1, n)
    star = torch.arange(1, n + 1)
    zero = torch.zeros_like(star)
    pick = torch.randint(0, len(w["ii"]), (2 * n,), generator=torch.Generator().manual_seed(n))
    w["ii"], w["jj"] = torch.cat([zero, star]), torch.cat([star, zero])
    w["targets"], w["weights"] = w["targets"][pick].contiguous(), w["weights"][pick].contiguous()
    r = oracle.ba.ba(*[w[k].double().numpy() for k in small.NAMES], w["ii"].numpy(), w["jj"].numpy(), 1, n + 1, 1, 1e-4,
                     0.1)
    d = {k: v.to(cuda) for k, v in w.items()}
    one = {k: v.clone() for k, v in d.items()}
    dx, dz, _ = droid_backends.ba(*[one[k] for k in small.NAMES], one["ii"], one["jj"], 1, n + 1, 1, 1e-4, 0.1, False)
    assert small.rel(dx, r.dx) < 1e-4 and small.rel(dz, r.dz) < 1e-4 and small.rel(one["disps"], r.disps) < 1e-4
    batch = backends.BABatch([dict(d, t0=1, t1=n + 1)], 1e-4, 0.1)
    batch.run(1)
    (dx, dz), = batch.results()
    assert small.rel(dx, r.dx) < 1e-4 and small.rel(dz, r.dz) < 1e-4 and small.rel(d["disps"], r.disps) < 1e-4
