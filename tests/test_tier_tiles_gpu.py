"""The tiered reference-rule assembly at the face counts where its tile sizes change, with lists of close pairs that
are full (k 30: every pair takes the reference's points) and nearly empty, against the face order.  Tolerance as in
test_mom_tiers_gpu.py."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 1e-6


@pytest.mark.parametrize("nf", [61, 120, 121, 441, 442, 986, 987, 2231, 2233, 4463, 4465])
@pytest.mark.parametrize("gq,k", [(3, 0.7), (3, 30.0), (4, 0.7), (4, 30.0), (5, 30.0)])
def test_tiers_at_the_steps_of_the_tiles(pkg, nf, gq, k):
    if gq == 5 and nf > 1000:
        pytest.skip("covered by gaussQR 3 and 4")
    u = pkg.utils
    v, f = pkg.meshes.icosphere(next(l for l in range(5) if 20 * 4 ** l >= nf))
    f = np.asarray(f)[:nf]  # open where the list ends
    used, inv = np.unique(f, return_inverse=True)
    V = torch.tensor(np.asarray(v)[used], dtype=torch.float32, device="cuda")
    F = torch.tensor(inv.reshape(-1, 3), dtype=torch.int32, device="cuda")
    edges, fei, _ = u.get_edge_unique(V, F)
    args = [V, F, u.compute_face_areas(V, F).contiguous(), u.compute_face_normals(V, F).contiguous(), fei,
            edges.shape[0], *u.get_gaussion_integration_points_and_weights(gq, device="cuda"),
            *u.get_gaussion_integration_points_and_weights(gq - 1, device="cuda"), k]
    ref = pkg.mesh_MOM_3d.assemble_Z_rwg(*args, order="faces")
    got = pkg.mesh_MOM_3d.assemble_Z_rwg(*args, order="tiers")
    assert (torch.linalg.norm(got - ref) / torch.linalg.norm(ref)).item() < TOL
