"""Restart lengths around the groups of steps that the preconditioned solver launches at once: captured and direct
launches do the same sums (bitwise), with the steps that max_iters allows.  Tolerance: the solver's own promise."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("restart", [1, 2, 7, 8, 9, 16, 17, 20, 128])
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_groups(pkg, restart, dtype):
    n, tol = 150, 1e-8
    g = torch.Generator(device="cuda").manual_seed(1)
    Z = torch.randn((n, n), generator=g, dtype=dtype, device="cuda") * (0.3 / n ** 0.5) + torch.eye(n, dtype=dtype, device="cuda")
    b = torch.randn(n, generator=g, dtype=torch.complex128, device="cuda")
    M = pkg.mesh_MOM_3d
    x, (i,) = M.pgmres(Z, b, restart=restart, tol=tol)
    y, (j,) = M.pgmres(Z, b, restart=restart, tol=tol, use_graph=False)
    assert torch.equal(x, y) and i == j and i["converged"]
    assert (torch.linalg.norm(b - Z.to(torch.complex128) @ x) / torch.linalg.norm(b)).item() <= 1.01 * tol
    for limit in (1, restart, restart + 1):
        if limit > 21:  # 1e-14 is reached in some forty steps
            continue
        _, (i,) = M.pgmres(Z, b, restart=restart, tol=1e-14, max_iters=limit)
        assert i["iterations"] == limit and not i["converged"] and i["restarts"] == -(-limit // restart)
