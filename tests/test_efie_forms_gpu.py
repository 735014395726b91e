"""The EFIE matrix on both sides of the lines between its two ways with separated pairs (each unordered pair once,
summed above the diagonal and mirrored, or on both sides of a given matrix; row by row): mesh sizes, faces in any order,
wavenumbers at which no, some and all pairs are too large for the first.  Reference: the row-by-row matrix
(faces_range), with the near pairs added.  Tolerance: that of test_efie_pairs_gpu.py."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf", [2399, 2400, 2431, 3000])
@pytest.mark.parametrize("kind", ["ordered", "runs of two", "shuffled"])
@pytest.mark.parametrize("k", [0.5, 7.0, 40.0])
def test_matrix_of_its_own(pkg, nf, kind, k):
    v, f = pkg.meshes.icosphere(4)
    f = np.asarray(f)[:nf]
    used, inv = np.unique(f, return_inverse=True)
    v, f = np.asarray(v)[used] * np.array([1.0, 0.8, 0.6]), inv.reshape(-1, 3)
    rng = np.random.default_rng(0)
    if kind == "shuffled":
        f = f[rng.permutation(nf)]
    if kind == "runs of two":
        f = f[np.concatenate([[2 * i, 2 * i + 1] for i in rng.permutation(nf // 2)] + [[nf - 1]] * (nf % 2)).astype(int)]
    V, F = torch.tensor(v, dtype=torch.float32, device="cuda"), torch.tensor(f, dtype=torch.int32, device="cuda")
    edges, fei, _ = pkg.utils.get_edge_unique(V, F)
    ne, M = edges.shape[0], pkg.mesh_MOM_3d
    pairs = M.near_pairs(F)
    ref = M.assemble_Z_rwg_sym(V, F, fei, ne, k, faces_range=(0, nf))
    L = pkg._lib
    L.call("mb_mom_sym_near_c64", L.ptr(V), V.shape[0], L.ptr(F), nf, L.ptr(fei), ne, L.ptr(pairs), pairs.shape[0], k,
           L.ptr(ref), L.stream_of(V))
    stale = torch.full((ne, ne), float("nan"), dtype=torch.complex64, device="cuda")  # what the new matrix is laid over
    del stale
    got = M.assemble_Z_rwg_sym(V, F, fei, ne, k, pairs=pairs)
    assert (torch.linalg.norm(got - ref) / torch.linalg.norm(ref)).item() < 1e-6
    twice = M.assemble_Z_rwg_sym(V, F, fei, ne, k, pairs=pairs, out=ref.clone())
    assert (torch.linalg.norm(twice - 2 * got) / torch.linalg.norm(ref)).item() < 2e-6
