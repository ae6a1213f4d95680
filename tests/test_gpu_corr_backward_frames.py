"""altcorr_backward packs only the frames that its edges can use: few edges over many frames, more
edges than frames, frames used on one side only, and radii on both sides of the tiled
kernel's limit, against the float64 oracle (1e-5 of the largest gradient in FP32); the
workspace sizes that follow; and the step down to the accumulators alone when the device has no
room for more.
"""

import ctypes

import pytest
import torch

import droid_backends
import oracle.corr as oc
from hislam2_b200 import _lib
from test_gpu_corr_backward import close, np64, problem

pytestmark = pytest.mark.gpu


def size(dt, B, N1, N2, C, hw, hw2, M, r):
    n = ctypes.c_size_t(0)
    assert _lib.load().hs2_altcorr_backward_call_workspace_size(dt, B, N1, N2, C, *hw, *hw2, M, r, ctypes.byref(n)) == 0
    return n.value


def check(f1, f2, crd, ii, jj, r, tol=1e-5):
    B, M, _, H, W = crd.shape
    g = torch.randn(B, M, 2 * r + 1, 2 * r + 1, H, W, generator=torch.Generator().manual_seed(5)).to(crd.device)
    g1, g2 = droid_backends.altcorr_backward(f1, f2, crd, ii, jj, g, r)
    r1, r2 = oc.altcorr_backward(np64(f1), np64(f2), np64(crd), ii.cpu().numpy(), jj.cpu().numpy(), np64(g), r)
    assert close(g1, r1, tol) and close(g2, r2, tol)


@pytest.mark.parametrize("B,N1,N2,M,r", [(2, 9, 1, 3, 3), (1, 1100, 1030, 3, 1), (2, 2, 3, 7, 4), (1, 3, 2, 4, 6),
                                         (1, 3, 2, 4, 7)])
def test_frames_in_use(cuda, B, N1, N2, M, r):
    f1, f2, crd, ii, jj = problem(B, N1, N2, 5, 6, 4, 3, M, N1 + r, cuda, torch.float32, 0.5)
    if N1 > 1024:            # the last frames, of the scan's second round, out of order
        ii = torch.tensor([N1 - 1, 3, 1025], device=cuda)
        jj = torch.tensor([1028, N2 - 1, 0], device=cuda)
    check(f1, f2, crd, ii, jj, r)


def test_workspace_sizes():
    frame = 128 * 43 * 77 * 4
    few, all_frames = (size(_lib.HS2_F32, 1, 300, 300, 128, (43, 77), (43, 77), M, 3) for M in (4, 5000))
    assert 16 * frame <= few < 17 * frame and 1200 * frame <= all_frames < 1201 * frame
    assert size(_lib.HS2_F32, 1, 300, 300, 128, (43, 77), (43, 77), 4, 7) == 0
    assert size(_lib.HS2_F32, 1, 300, 300, 64, (43, 77), (43, 77), 4, 3) == 0


def test_no_room_for_the_tiles(cuda, monkeypatch):
    f1, f2, crd, ii, jj = problem(1, 4, 4, 9, 10, 9, 10, 5, 3, cuda, torch.float32, 0.5)
    most, empty, refused = f1.numel() * 4, torch.empty, []

    def tight(*shape, **kw):
        if kw.get("dtype") == torch.uint8 and shape[0] > most:
            refused.append(shape[0])
            raise torch.cuda.OutOfMemoryError("no room")
        return empty(*shape, **kw)

    monkeypatch.setattr(torch, "empty", tight)
    check(f1, f2, crd, ii, jj, 3)
    assert len(refused) == 1
