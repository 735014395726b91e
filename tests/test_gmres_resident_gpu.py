"""The resident restart cycle of mb_gmres_* at the sizes where its row ranges, split rows and
vector paths change, against a dense FP64 solve.

Tolerances: the solver promises a true residual below tol (checked in FP64 against the
matrix it was given); the solution of these systems (condition number below 10) is then
within 10 tol of the dense one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _system(n, dtype, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    A = torch.randn((n, n), generator=g, dtype=dtype, device="cuda") * (0.3 / n ** 0.5)
    A += torch.eye(n, dtype=dtype, device="cuda")
    wide = torch.complex128 if dtype.is_complex else torch.float64
    return A, torch.randn(n, generator=g, dtype=wide, device="cuda")


# one row; fewer rows than a block's 8; odd (no vector loads) and even; 151 workers of 8 rows and one more
# row; more rows than warps per block; a vector that no longer fits beside the basis
@pytest.mark.parametrize("n", [1, 2, 7, 9, 33, 1207, 1208, 1209, 4833, 9000])
@pytest.mark.parametrize("dtype", [torch.complex64, torch.float32, torch.float64])
@pytest.mark.parametrize("restart", [5, 60])
def test_resident_cycle_solves(pkg, n, dtype, restart):
    if n > 2000 and (restart == 5 or dtype == torch.float64):
        pytest.skip("covered by the smaller sizes")
    A, b = _system(n, dtype)
    tol = 1e-9
    solve = pkg.mesh_MOM_3d.gmres if dtype.is_complex else pkg.mesh_MOM_3d.gmres_real
    x, (info,) = solve(A, b, restart=restart, tol=tol)
    W = A.to(b.dtype)
    assert info["converged"] and info["rel_residual"] <= tol
    assert (torch.linalg.norm(b - W @ x) / torch.linalg.norm(b)).item() <= 1.01 * tol
    ref = torch.linalg.solve(W, b)
    assert (torch.linalg.norm(x - ref) / torch.linalg.norm(ref)).item() < 10 * tol


def test_limits_and_starting_values(pkg):
    A, b = _system(300, torch.complex64, 1)
    gm = pkg.mesh_MOM_3d.gmres
    x, (i,) = gm(A, b, restart=128, tol=1e-8)
    assert i["restarts"] >= 1 and i["converged"]
    _, (i,) = gm(A, b, restart=10, tol=1e-8, max_iters=3)  # stops at the limit, reports the residual reached
    assert i["iterations"] == 3 and not i["converged"] and 1e-8 < i["rel_residual"] < 1
    _, (i,) = gm(A, b, x0=x, tol=1e-7)  # already solved: no step
    assert i["iterations"] == 0 and i["converged"]
    x0, (i,) = gm(A, torch.zeros_like(b), tol=1e-8)
    assert i["converged"] and i["iterations"] == 0 and not x0.abs().any()
    many, infos = gm(A, torch.stack((b, 2j * b), 1), tol=1e-8)
    assert len(infos) == 2 and torch.allclose(many[:, 1], 2j * many[:, 0], rtol=0, atol=1e-6)
    eye = torch.eye(300, dtype=torch.complex64, device="cuda")
    _, (i,) = gm(eye, b, tol=1e-8)  # invariant after one step but for the FP32 rounding of the vector
    assert i["converged"] and i["iterations"] <= 3
