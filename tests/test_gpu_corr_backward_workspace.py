"""altcorr_backward with workspaces that start at any multiple of its accumulators' 4 bytes, and
corr_lookup_backward, which refuses one off its 16-byte boundary.  Gradients against the float64 oracle:
1e-5 of the largest in FP32, half the type's spacing on top in FP16.
"""

import ctypes

import pytest
import torch

import oracle.corr as oc
from hislam2_b200 import _lib, backends
from test_gpu_corr_backward import close, np64, problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.float16, 1e-5 + 2 ** -11)], ids=["f32", "f16"])
@pytest.mark.parametrize("offset", [0, 4, 8, 12])
def test_any_alignment(cuda, offset, dtype, tol):
    H, W, H2, W2, r, M = 9, 10, 5, 6, 3, 4
    f1, f2, crd, ii, jj = problem(1, 3, 2, H, W, H2, W2, M, 1, cuda, dtype, 0.5)
    g = torch.randn(1, M, 2 * r + 1, 2 * r + 1, H, W, generator=torch.Generator().manual_seed(5)).to(cuda)
    lib, n, p = _lib.load(), ctypes.c_size_t(0), backends._ptr
    dt = backends._DTYPES[dtype]
    assert lib.hs2_altcorr_backward_workspace_size(dt, 1, 3, 2, 128, H, W, H2, W2, ctypes.byref(n)) == 0
    ws = torch.empty(n.value + 16, dtype=torch.uint8, device=cuda)
    g1, g2 = torch.empty_like(f1), torch.empty_like(f2)
    info = torch.zeros(1, dtype=torch.int32, device=cuda)
    rc = lib.hs2_altcorr_backward(p(f1), p(f2), dt, 1, 3, 2, 128, H, W, H2, W2, p(crd), p(ii), p(jj), M, p(g), r, 1.0,
                                  p(g1), p(g2), p(info), ctypes.c_void_p(ws.data_ptr() + offset), n.value,
                                  backends._stream(cuda))
    assert rc == 0 and int(info.item()) == 0
    r1, r2 = oc.altcorr_backward(np64(f1), np64(f2), np64(crd), ii.cpu().numpy(), jj.cpu().numpy(), np64(g), r)
    assert close(g1, r1, tol) and close(g2, r2, tol)


def test_lookup_backward_refuses_a_workspace_off_its_boundary(cuda):
    f = torch.randn(1, 128, 8, 8, device=cuda)
    crd, g = torch.zeros(1, 8, 8, 2, device=cuda), torch.zeros(1, 49, 8, 8, device=cuda)
    lib, n, p = _lib.load(), ctypes.c_size_t(0), backends._ptr
    assert lib.hs2_corr_lookup_backward_workspace_size(_lib.HS2_F32, 1, 128, 8, 8, 1, 3, ctypes.byref(n)) == 0
    ws = torch.empty(n.value + 16, dtype=torch.uint8, device=cuda)
    rc = lib.hs2_corr_lookup_backward(p(f), p(f), _lib.HS2_F32, 1, 128, 8, 8, p(crd), p(g), 1, 3, 1.0,
                                      p(torch.empty_like(f)), p(torch.empty_like(f)),
                                      ctypes.c_void_p(ws.data_ptr() + 8), n.value, backends._stream(cuda))
    assert rc == _lib.HS2_ERR_WORKSPACE
