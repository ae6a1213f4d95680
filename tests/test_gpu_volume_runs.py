"""corr_volume at the sizes where its output runs can go wrong: widths on both sides of a 16-column
piece and of the kernel's staging limits, odd heights, fewer levels, planes smaller than a
16-byte chunk, one pair (units split by image rows) and many, live rows that end inside a
warp, pairs with an index out of range among valid ones.

Level 0 against a float64 product (FP16 2^-10, BF16 2^-7 of the largest value: one rounding of
an FP32 sum); every pooled level equals avg_pool2d of the level above bit for bit; guard bands
around the outputs stay untouched.
"""

import ctypes

import pytest
import torch
import torch.nn.functional as F

from hislam2_b200 import _lib, backends

pytestmark = pytest.mark.gpu


def guarded(fmap, ii, jj, levels, precision):
    """hs2_corr_volume into buffers with 64 sentinel elements on either side."""
    K, C, H, W = fmap.shape
    E, dev = ii.numel(), fmap.device
    raw, out = [], []
    for l in range(levels):
        n = E * H * W * (H >> l) * (W >> l)
        buf = torch.full((n + 128,), 7.0, dtype=fmap.dtype, device=dev)
        raw.append((buf, n))
        out.append(buf[64:64 + n].view(E, H, W, H >> l, W >> l))
    prec = {"native": _lib.HS2_CV_NATIVE, "e4m3": _lib.HS2_CV_E4M3}[precision]
    dt = backends._DTYPES[fmap.dtype]
    lib, nbytes = _lib.load(), ctypes.c_size_t(0)
    assert lib.hs2_corr_volume_workspace_size(K, K, C, H, W, dt, prec, ctypes.byref(nbytes)) == 0
    ws = torch.empty(nbytes.value, dtype=torch.uint8, device=dev)
    info = torch.zeros(1, dtype=torch.int32, device=dev)
    ptrs = (ctypes.c_void_p * 4)(*[o.data_ptr() for o in out] + [0] * (4 - levels))
    rc = lib.hs2_corr_volume(backends._ptr(fmap), K, backends._ptr(fmap), K, C, H, W, dt, backends._ptr(ii),
                             backends._ptr(jj), E, prec, levels, ptrs, backends._ptr(info), backends._ptr(ws),
                             nbytes.value, backends._stream(dev))
    assert rc == 0
    torch.cuda.synchronize()
    for buf, n in raw:
        assert (buf[:64] == 7).all() and (buf[64 + n:] == 7).all()
    return out, int(info.item())


@pytest.mark.parametrize("precision", ["native", "e4m3"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["f16", "bf16"])
@pytest.mark.parametrize("H,W,E,levels", [(1, 1, 3, 4), (3, 2, 5, 3), (8, 15, 2, 4), (9, 16, 1, 4), (17, 17, 2, 4),
                                          (24, 33, 1, 4), (7, 64, 3, 2), (33, 65, 1, 4), (10, 79, 2, 4), (41, 80, 1, 4),
                                          (6, 81, 3, 4), (19, 96, 1, 4), (43, 77, 1, 1)])
def test_volume_runs(cuda, H, W, E, levels, dtype, precision):
    g = torch.Generator().manual_seed(H * W)
    f = (torch.randn(3, 128, H, W, generator=g) / 128 ** 0.5).to(dtype).to(cuda)
    ii = torch.randint(0, 3, (E,), generator=g).to(cuda)
    jj = torch.randint(0, 3, (E,), generator=g).to(cuda)
    out, bits = guarded(f, ii, jj, levels, precision)
    assert bits == 0
    a = f[ii].double().flatten(2) / 4
    b = f[jj].double().flatten(2) / 4
    ref = (a.transpose(1, 2) @ b).view(E, H, W, H, W)
    tol = 0.12 if precision == "e4m3" else 2.0 ** -10 if dtype == torch.float16 else 2.0 ** -7
    assert (out[0].double() - ref).abs().max() <= tol * ref.abs().max()
    for l in range(1, levels):
        h, w = H >> (l - 1), W >> (l - 1)
        if out[l].numel():
            up = F.avg_pool2d(out[l - 1].reshape(E * H * W, 1, h, w), 2, stride=2)
            assert torch.equal(up.reshape(out[l].shape), out[l]), l


def test_volume_bad_pairs_between_good_ones(cuda):
    f = torch.randn(2, 128, 11, 13, device=cuda).half()
    good, _ = guarded(f, torch.tensor([0, 1], device=cuda), torch.tensor([1, 1], device=cuda), 4, "native")
    out, bits = guarded(f, torch.tensor([0, 5, 1, -1], device=cuda), torch.tensor([1, 0, 1, 1], device=cuda), 4, "native")
    assert bits & _lib.HS2_DEV_BAD_INDEX
    for a, b in zip(good, out):
        assert torch.equal(a, b[[0, 2]])
        assert (b[[1, 3]] == 7).all()
