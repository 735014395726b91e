"""float64 systems of entries near the ends of the range, where |h|^2 leaves it and |h| does not: the Givens
rotation's length has to come from the values.  The matrix is s times one that GMRES solves in a
step (a multiple of the identity) or a few.  Tolerance: the solver's own promise."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-170, 1e-157, 1.0, 1e157, 1e160])
def test_scaled_identity(pkg, scale):
    n = 64
    A = scale * torch.eye(n, dtype=torch.float64, device="cuda")
    b = torch.randn(n, generator=torch.Generator(device="cuda").manual_seed(2), dtype=torch.float64, device="cuda")
    x, (info,) = pkg.mesh_MOM_3d.gmres_real(A, b, tol=1e-10)
    assert info["converged"] and info["iterations"] <= 3
    assert (torch.linalg.norm(x * scale - b) / torch.linalg.norm(b)).item() <= 1.01e-10


@pytest.mark.parametrize("scale", [1e-140, 1e140])
def test_scaled_system(pkg, scale):
    n = 200
    g = torch.Generator(device="cuda").manual_seed(4)
    A = torch.eye(n, dtype=torch.float64, device="cuda")
    A += torch.randn((n, n), generator=g, dtype=torch.float64, device="cuda") * (0.3 / n ** 0.5)
    b = torch.randn(n, generator=g, dtype=torch.float64, device="cuda")
    x, (info,) = pkg.mesh_MOM_3d.gmres_real(scale * A, b, tol=1e-10)
    _, (one,) = pkg.mesh_MOM_3d.gmres_real(A, b, tol=1e-10)
    assert info["converged"] and abs(info["iterations"] - one["iterations"]) <= 1
    assert (torch.linalg.norm(A @ (x * scale) - b) / torch.linalg.norm(b)).item() <= 1.01e-10
