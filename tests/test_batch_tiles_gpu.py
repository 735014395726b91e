"""Batched reference-rule matrices against each mesh's own, evaluated at the reference's points (the face order), over
the batch's choice of kernel and tiles: meshes below and above 256 faces, gaussQR 3 at few and many face pairs,
the tile sizes' steps, meshes that end inside a tile.  Tolerance as in test_mom_tiers_gpu.py."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 1e-6


def _mesh(pkg, nf):
    """The first nf faces of an icosphere, squeezed (open where they end)."""
    v, f = pkg.meshes.icosphere(next(l for l in range(5) if 20 * 4 ** l >= nf))
    f = np.asarray(f)[:nf]
    used, inv = np.unique(f, return_inverse=True)
    return np.asarray(v)[used] * np.array([1.0, 0.8, 0.9]), inv.reshape(-1, 3).astype(np.int32)


@pytest.mark.parametrize("faces", [(20,), (20, 7, 80, 33), (255, 80), (256, 80, 9), (300, 20, 257), (640, 320, 90), (1111, 61)])
@pytest.mark.parametrize("gq", [2, 3, 4, 5])
def test_batch_equals_the_meshes(pkg, faces, gq):
    if gq == 5 and max(faces) > 640:
        pytest.skip("covered by gaussQR 4")
    u = pkg.utils
    meshes, ks = [_mesh(pkg, n) for n in faces], [0.7 + 2.0 * i for i in range(len(faces))]
    B = pkg.batch.MeshBatch(meshes, ks, device="cuda:0", formulation="cfie_ref", gaussQR=gq)
    z = B.assemble(out=torch.full((B.z_size,), 3.0, dtype=torch.complex64, device="cuda"))
    rules = [*u.get_gaussion_integration_points_and_weights(gq, device="cuda"),
             *u.get_gaussion_integration_points_and_weights(gq - 1, device="cuda")]
    for i, (v, f) in enumerate(meshes):
        V, F = torch.tensor(v, dtype=torch.float32, device="cuda"), torch.tensor(f, device="cuda")
        edges, fei, _ = u.get_edge_unique(V, F)
        ref = pkg.mesh_MOM_3d.assemble_Z_rwg(V, F, u.compute_face_areas(V, F).contiguous(),
                                             u.compute_face_normals(V, F).contiguous(), fei, edges.shape[0], *rules,
                                             ks[i], order="faces")
        got = B.z_block(z, i)
        assert (torch.linalg.norm(got - ref) / torch.linalg.norm(ref)).item() < TOL


def test_tile_sizes_are_what_the_kernels_take(pkg):
    for pairs in [0, 1, 400, 14591, 14592, 194559, 194560, 972799, 972800, 4980735, 4980736, 19922943, 19922944, 10 ** 12]:
        t = [ctypes.c_int32() for _ in range(3)]
        pkg._lib.call("mb_mom_tier_tiles", pairs, *(ctypes.byref(x) for x in t))
        rows, tp, tq = (x.value for x in t)
        assert 1 <= rows <= 32 and 1 <= tp <= 256 and 1 <= tq <= 128 and tq & (tq - 1) == 0 and tp * tq <= 1024
