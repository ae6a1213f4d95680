"""corr_volume into levels that start at any element: the four levels one after the other in one
buffer whose first element lies at each of the eight 2-byte phases of a 16-byte chunk, so that
every level meets odd and even phases.  The values are those of separately allocated levels bit
for bit, and the elements before and behind the levels stay as they were.
"""

import ctypes

import pytest
import torch

from hislam2_b200 import _lib, backends

pytestmark = pytest.mark.gpu


def volume_at(fmap, ii, jj, out, precision):
    K, C, H, W = fmap.shape
    dt, lib, nbytes = backends._DTYPES[fmap.dtype], _lib.load(), ctypes.c_size_t(0)
    assert lib.hs2_corr_volume_workspace_size(K, K, C, H, W, dt, precision, ctypes.byref(nbytes)) == 0
    ws = torch.empty(nbytes.value, dtype=torch.uint8, device=fmap.device)
    info = torch.zeros(1, dtype=torch.int32, device=fmap.device)
    ptrs = (ctypes.c_void_p * 4)(*[o.data_ptr() for o in out])
    assert lib.hs2_corr_volume(backends._ptr(fmap), K, backends._ptr(fmap), K, C, H, W, dt, backends._ptr(ii),
                               backends._ptr(jj), ii.numel(), precision, 4, ptrs, backends._ptr(info),
                               backends._ptr(ws), nbytes.value, backends._stream(fmap.device)) == 0
    torch.cuda.synchronize()
    assert int(info.item()) == 0


@pytest.mark.parametrize("precision", [_lib.HS2_CV_NATIVE, _lib.HS2_CV_E4M3], ids=["native", "e4m3"])
@pytest.mark.parametrize("H,W,E", [(9, 11, 3), (16, 33, 1), (17, 64, 2), (8, 81, 1)])
@pytest.mark.parametrize("phase", range(8))
def test_levels_in_one_buffer(cuda, H, W, E, phase, precision):
    g = torch.Generator().manual_seed(H * W)
    f = (torch.randn(3, 128, H, W, generator=g) / 128 ** 0.5).half().to(cuda)
    ii, jj = (torch.randint(0, 3, (E,), generator=g).to(cuda) for _ in range(2))
    shapes = [(E, H, W, H >> l, W >> l) for l in range(4)]
    apart = [torch.empty(s, dtype=f.dtype, device=cuda) for s in shapes]
    volume_at(f, ii, jj, apart, precision)
    sizes = [o.numel() for o in apart]
    buf = torch.full((64 + phase + sum(sizes) + 64,), 7.0, dtype=f.dtype, device=cuda)
    assert buf.data_ptr() % 16 == 0
    at, placed = 64 + phase, []
    for s, n in zip(shapes, sizes):
        placed.append(buf[at:at + n].view(s))
        at += n
    volume_at(f, ii, jj, placed, precision)
    for a, b in zip(apart, placed):
        assert torch.equal(a, b)
    assert (buf[:64 + phase] == 7).all() and (buf[at:] == 7).all()
