"""The instances of mb_gmres_* that test_gmres_resident_gpu.py does not reach: the resident cycle whose basis vector no
longer fits beside the basis in shared memory (at restart 128; at 60 it fits up to the largest system), and, above
12288 unknowns, the launch per operation.  Tolerance: the solver's own promise, checked in FP64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,restart,dtype", [
    (10800, 128, torch.complex64), (10801, 128, torch.complex64), (10800, 128, torch.float32), (10803, 128, torch.float32),
    (7700, 128, torch.float64), (7701, 128, torch.float64),
    (12288, 20, torch.complex64), (12289, 20, torch.complex64), (12289, 20, torch.float32), (12289, 20, torch.float64)])
def test_large_systems(pkg, n, restart, dtype):
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn((n, n), generator=g, dtype=dtype, device="cuda").mul_(0.5 / n ** 0.5)
    A.diagonal().add_(1)
    b = torch.randn(n, generator=g, dtype=torch.complex128 if dtype.is_complex else torch.float64, device="cuda")
    solve = pkg.mesh_MOM_3d.gmres if dtype.is_complex else pkg.mesh_MOM_3d.gmres_real
    x, (info,) = solve(A, b, restart=restart, tol=1e-10)
    assert info["converged"] and info["rel_residual"] <= 1e-10
    r = b.clone()
    for i in range(0, n, 2048):  # by parts: the whole matrix in FP64 is not needed
        r[i:i + 2048] -= A[i:i + 2048].to(b.dtype) @ x
    assert (torch.linalg.norm(r) / torch.linalg.norm(b)).item() <= 1.01e-10
