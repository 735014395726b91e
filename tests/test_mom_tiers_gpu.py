"""The tiered reference-rule assembly (``order="tiers"``) against the face order, which evaluates the
reference's points on every pair, and by distance against float64.

Tolerance: both orders evaluate the close pairs, which make up most of the norm and of the
FP32 error (1e-6 .. 2e-6 of the float64 matrix on the sphere of slivers, 3e-7 .. 6e-7 on the
others), with the same arithmetic; on the others a tier's rule is off by at most 2e-6 of an
entry, and those entries are a small part of the norm: 1e-6."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 1e-6


@pytest.fixture(scope="module")
def pkg():
    import importlib

    return importlib.import_module("mesh-ferrofluid_gb300")


def _uv(lat, lon):
    th, ph = np.pi * np.arange(1, lat) / lat, 2 * np.pi * np.arange(lon) / lon
    ring = np.stack((np.outer(np.sin(th), np.cos(ph)), np.outer(np.sin(th), np.sin(ph)),
                     np.outer(np.cos(th), np.ones(lon))), -1).reshape(-1, 3)
    v = np.concatenate(([[0, 0, 1.0]], ring, [[0, 0, -1.0]]))
    n, f = lat - 1, []
    for j in range(lon):
        k = (j + 1) % lon
        f.append((0, 1 + j, 1 + k))
        for i in range(n - 1):
            a, b = 1 + i * lon, 1 + (i + 1) * lon
            f += [(a + j, b + j, b + k), (a + j, b + k, a + k)]
        f.append((1 + (n - 1) * lon + j, v.shape[0] - 1, 1 + (n - 1) * lon + k))
    return v, np.asarray(f, np.int32)


def _setup(pkg, v, f, gq, dtype):
    u = pkg.utils
    verts = torch.tensor(np.asarray(v), dtype=torch.float32, device="cuda").to(dtype)
    faces = torch.tensor(np.asarray(f), dtype=torch.int32, device="cuda")
    edges, fei, _ = u.get_edge_unique(verts, faces)
    r32 = [*u.get_gaussion_integration_points_and_weights(gq, device="cuda"),
           *u.get_gaussion_integration_points_and_weights(gq - 1, device="cuda")]
    return [verts, faces, u.compute_face_areas(verts, faces).contiguous(),
            u.compute_face_normals(verts, faces).contiguous(), fei, edges.shape[0], *[t.to(dtype) for t in r32]]


def _rel(a, b):
    return (torch.linalg.norm(a.to(torch.complex128) - b) / torch.linalg.norm(b)).item()


# faces below, at and above the tile sizes (14, 16, 64, 128 faces; 8 and 32 rows), a sphere of slivers
@pytest.mark.parametrize("mesh", [("ico", 0), ("ico", 1), ("uv", 5, 8), ("uv", 9, 8), ("uv", 17, 9), ("uv", 12, 31),
                                  ("uv", 25, 54), ("uv", 4, 97)])
@pytest.mark.parametrize("gq,k", [(3, 0.3), (4, 0.3), (4, 2.5), (4, 12.0), (5, 2.5)])
def test_tiers_equal_the_face_order(pkg, mesh, gq, k):
    v, f = pkg.meshes.icosphere(mesh[1]) if mesh[0] == "ico" else _uv(*mesh[1:])
    if f.shape[0] > 1000 and gq == 5:
        pytest.skip("covered by gaussQR 4")
    a32 = _setup(pkg, v, f, gq, torch.float32)
    ref = pkg.mesh_MOM_3d.assemble_Z_rwg(*a32, k, order="faces").to(torch.complex128)
    Z = pkg.mesh_MOM_3d.assemble_Z_rwg(*a32, k, order="tiers")
    assert _rel(Z, ref) < TOL
    auto = pkg.mesh_MOM_3d.assemble_Z_rwg(*a32, k, out=Z.clone())  # accumulates
    assert _rel(auto, 2 * ref) < TOL


def test_every_band_of_distances_is_as_accurate_as_the_edge_order(pkg):
    """Entry errors by edge distance, against the float64 matrix: at most 1.5 times those of the
    1296 points (the bands nearest the change of rule have the few entries at its tolerance)."""
    v, f = pkg.meshes.ellipsoid(3, jitter=0.01, seed=3)
    a64, a32 = (_setup(pkg, v, f, 4, dt) for dt in (torch.float64, torch.float32))
    ref = pkg.mesh_MOM_3d.assemble_Z_rwg(*a64, 1.5)
    Z = {o: pkg.mesh_MOM_3d.assemble_Z_rwg(*a32, 1.5, order=o) for o in ("tiers", "edges")}
    edges, _, _ = pkg.utils.get_edge_unique(a64[0], a64[1])
    mid = a64[0][edges.long()].mean(1)
    R = torch.cdist(mid, mid)
    for lo, hi in ((0, 0.3), (0.3, 0.6), (0.6, 1.0), (1.0, 3.0)):
        m = (R >= lo) & (R < hi)
        err = {o: torch.linalg.norm(z[m].to(torch.complex128) - ref[m]).item() for o, z in Z.items()}
        assert err["tiers"] < 1.5 * err["edges"], (lo, hi, err)


def test_other_rules_and_normals_take_the_reference_points(pkg):
    """Nodes that are not Gauss-Legendre and normals that are not perpendicular to their faces:
    every pair concerned keeps the rule given (equal to the face order)."""
    v, f = _uv(14, 16)
    args = _setup(pkg, v, f, 4, torch.float32)
    for change in ("rule", "normal"):
        b = [t.clone() if torch.is_tensor(t) else t for t in args]
        if change == "rule":
            b[6] = b[6] * 0.9 + 0.05
        else:
            b[3] = torch.nn.functional.normalize(b[3] + 0.1, dim=-1).contiguous()
        ref = pkg.mesh_MOM_3d.assemble_Z_rwg(*b, 0.5, order="faces")
        assert _rel(pkg.mesh_MOM_3d.assemble_Z_rwg(*b, 0.5, order="tiers"), ref.to(torch.complex128)) < 5e-7


def test_open_and_branching_meshes(pkg):
    """Boundary edges (one face) and an edge with three faces."""
    v = np.array([[0, 0, 0], [1, 0, 0], [0.5, 0.9, 0], [0.5, 0.3, 0.8], [0.5, -0.6, -0.7], [6, 0, 0], [6.3, 0, 0],
                  [6.1, 0.3, 0.1]], float) * 0.2
    f = np.array([[0, 1, 2], [0, 1, 3], [1, 0, 4], [5, 6, 7]], np.int32)
    ref = pkg.mesh_MOM_3d.assemble_Z_rwg(*_setup(pkg, v, f, 4, torch.float64), 1.0)
    assert _rel(pkg.mesh_MOM_3d.assemble_Z_rwg(*_setup(pkg, v, f, 4, torch.float32), 1.0), ref) < TOL


def test_no_faces(pkg):
    a = _setup(pkg, np.eye(3), np.array([[0, 1, 2]], np.int32), 4, torch.float32)
    z = torch.zeros(0, dtype=torch.int32, device="cuda")
    Z = pkg.mesh_MOM_3d.assemble_Z_rwg(a[0], z.reshape(0, 3), a[2][:0], a[3][:0], z, 2, *a[6:], 1.0)
    assert Z.shape == (2, 2) and not Z.abs().any()
