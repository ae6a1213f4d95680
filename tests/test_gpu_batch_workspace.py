"""The batched solver on workspaces that start at any multiple of 8 bytes: the same poses, disparities
and increments as on one of its own, to the bar of the batched tests (1e-4 of the largest
magnitude; the sums are atomic, in any order).
"""

import ctypes

import pytest
import torch

from hislam2_b200 import _lib, backends
from test_gpu_batch_gram import rel, star

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 8, 248])
def test_any_alignment(cuda, offset):
    out = []
    for at in (None, offset):
        ws = [{k: (v.to(cuda) if torch.is_tensor(v) else v) for k, v in star(K, h, w, K).items()}
              for K, h, w in [(5, 7, 11), (16, 6, 13), (43, 5, 7)]]
        plan = backends.BABatch(ws, 1e-4, 0.1)
        if at is not None:
            n, grid = plan.ws.numel(), ctypes.c_int(0)
            raw = torch.empty(n + 512, dtype=torch.uint8, device=cuda)
            plan.ws = raw[-raw.data_ptr() % 256 + at:][:n]
            _lib.check(_lib.load().hs2_ba_batch_prepare(plan._arr, len(ws), 4, 0, backends._ptr(plan.ws), n,
                                                        ctypes.byref(grid), backends._stream(cuda)), "prepare")
            plan.grid = grid.value
        plan.run(2)
        out.append([t for (dx, dz), w in zip(plan.results(), ws) for t in (dx, dz, w["poses"], w["disps"])])
    for a, b in zip(*out):
        assert torch.isfinite(b).all() and rel(b, a.double().cpu().numpy()) < 1e-4
