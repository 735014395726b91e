"""mb_gmres_c64 with b, or the workspace, on an 8-byte but not a 16-byte boundary (through the C ABI: a
caller's buffer of doubles, entered at an odd place).  Such calls run as launches; the resident
cycle takes 16-byte boundaries only.  Tolerance: the solver's own promise, checked in FP64."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,restart", [(33, 10), (300, 50)])
@pytest.mark.parametrize("shifted", ["b", "workspace", "both", "neither"])
def test_eight_byte_boundaries(pkg, n, restart, shifted):
    L = pkg._lib
    g = torch.Generator(device="cuda").manual_seed(n)
    Z = torch.randn((n, n), generator=g, dtype=torch.complex64, device="cuda") * (0.3 / n ** 0.5)
    Z += torch.eye(n, dtype=torch.complex64, device="cuda")
    need = int(L.load().mb_gmres_workspace_bytes(n, restart))
    ws = torch.empty(need + 8, dtype=torch.uint8, device="cuda")
    o = 8 if shifted in ("workspace", "both") else 0
    buf = torch.randn(2 * n + 1, generator=g, dtype=torch.float64, device="cuda")
    ob = 1 if shifted in ("b", "both") else 0
    b = buf[ob:ob + 2 * n]
    x = torch.zeros(n, dtype=torch.complex128, device="cuda")
    assert ws.data_ptr() % 16 == 0 and buf.data_ptr() % 16 == 0
    info, tol = L.GmresInfo(), 1e-9
    L.call("mb_gmres_c64", L.ptr(Z), n, L.ptr(b), L.ptr(x), restart, 500, tol, ctypes.c_void_p(ws.data_ptr() + o), need,
           ctypes.byref(info), L.stream_of(Z))
    rhs = torch.complex(b[0::2], b[1::2])
    assert info.status == 0
    assert (torch.linalg.norm(rhs - Z.to(torch.complex128) @ x) / torch.linalg.norm(rhs)).item() <= 1.01 * tol
