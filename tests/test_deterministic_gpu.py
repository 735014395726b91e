"""Under torch.use_deterministic_algorithms the default float32 CFIE matrix repeats bit for bit (the edge order's two
additions per entry), as the orders "edges" and "gather" always do."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_default_order_repeats(pkg):
    u, M = pkg.utils, pkg.mesh_MOM_3d
    v, f = pkg.meshes.icosphere(3)
    V, F = torch.tensor(v, dtype=torch.float32, device="cuda"), torch.tensor(f, dtype=torch.int32, device="cuda")
    edges, fei, _ = u.get_edge_unique(V, F)
    args = [V, F, u.compute_face_areas(V, F).contiguous(), u.compute_face_normals(V, F).contiguous(), fei, edges.shape[0],
            *u.get_gaussion_integration_points_and_weights(4, device="cuda"),
            *u.get_gaussion_integration_points_and_weights(3, device="cuda"), 2.0]
    ref = M.assemble_Z_rwg(*args, order="edges")
    try:
        torch.use_deterministic_algorithms(True)
        runs = [M.assemble_Z_rwg(*args) for _ in range(5)]
    finally:
        torch.use_deterministic_algorithms(False)
    assert all(torch.equal(z, ref) for z in runs)
    gather = [M.assemble_Z_rwg(*args, order="gather") for _ in range(3)]
    assert all(torch.equal(z, gather[0]) for z in gather)
