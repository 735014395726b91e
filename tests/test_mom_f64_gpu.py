"""The FP64 reference-rule entries against the float64 oracle.

Tolerance: both are FP64 sums of the same points; an entry's rounding is a few 1e-15 of it, and
the phase k R adds its own rounding, k R times 2e-16, on both sides; between close faces an edge length over their distance (up to about 10 here) comes
on top: 3e-14 (1 + k R_max)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pkg():
    import importlib

    return importlib.import_module("mesh-ferrofluid_gb300")


def _mesh(pkg, name):
    v, f = pkg.meshes.icosphere(1 if name != "ico0" else 0)
    v, f = np.asarray(v, np.float64), np.asarray(f, np.int32)
    if name == "squeezed":  # slivers, and close faces that share nothing
        v = v * np.array([1.0, 0.7, 0.05])
    if name == "two":  # two bodies a few edges apart, and neither a multiple of a warp
        v = np.concatenate((v, 0.2 * v + np.array([0.0, 0.0, 1.5])))
        f = np.concatenate((f, f + v.shape[0] // 2))[:-9]
    return v, f


# source rules with a kernel of their own (1, 4, 9, 16 points) and the first without (25); column counts
# of 60, 240 and 453; wavenumbers from a phase that never turns to several hundred turns of the table
@pytest.mark.parametrize("name,gq,k", [("ico0", 2, 0.3), ("ico0", 5, 2.0), ("ico0", 6, 2.0), ("squeezed", 2, 5.0),
                                       ("squeezed", 3, 0.05), ("squeezed", 4, 400.0), ("two", 2, 3.0), ("two", 3, 3.0),
                                       ("two", 4, 1.0), ("two", 5, 40.0)])
def test_f64_entries(pkg, oracle, name, gq, k):
    u = pkg.utils
    v_np, f_np = _mesh(pkg, name)
    v = torch.tensor(v_np, device="cuda")
    f = torch.tensor(f_np, device="cuda")
    a, n = u.compute_face_areas(v, f).contiguous(), u.compute_face_normals(v, f).contiguous()
    rules = [*u.get_gaussion_integration_points_and_weights(gq, device="cuda", dtype=torch.float64),
             *u.get_gaussion_integration_points_and_weights(gq - 1, device="cuda", dtype=torch.float64)]
    h = lambda t: t.cpu().numpy()  # noqa: E731
    ref = oracle.mom_zmat_fe(v_np, f_np, h(a), h(n), *(h(t) for t in rules), k)
    ncol = 3 * f_np.shape[0]
    tol = 3e-14 * (1 + k * 2 * np.abs(v_np).max())
    fei = torch.arange(ncol, dtype=torch.int32, device="cuda").reshape(-1, 3)  # an edge of its own for each column
    z = pkg.mesh_MOM_3d.assemble_Z_rwg(v, f, a, n, fei, ncol, *rules, k)
    assert np.linalg.norm(h(z) - ref) <= tol * np.linalg.norm(ref)
    # a range of rows that starts inside a face and is no multiple of a block's rows
    r0, r1 = 7, ncol - 4
    z = pkg.mesh_MOM_3d.assemble_Z_rwg(v, f, a, n, fei, ncol, *rules, k, rows=(r0, r1))
    assert np.linalg.norm(h(z)[r0:r1] - ref[r0:r1]) <= tol * np.linalg.norm(ref)
    assert not h(z)[:r0].any() and not h(z)[r1:].any()
