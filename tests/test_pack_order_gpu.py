"""Packing of stored FP32 panels on both sides of the choice of its kernel: the mesh's size, the order of its faces and of
its vertices, more vertices than the rows' shared memory holds.  Reference: index_add in FP64; tolerance as in
test_vertex_slots_gpu.py (up to 36 FP32 terms an entry, in another order)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 1e-6


@pytest.mark.parametrize("nf,nv_extra", [(1, 0), (9, 0), (33, 5), (640, 0), (2499, 0), (2500, 0), (2600, 20000)])
@pytest.mark.parametrize("kind", ["ordered", "faces shuffled", "vertices shuffled", "corners apart"])
def test_pack(pkg, nf, nv_extra, kind):
    v, f = pkg.meshes.icosphere(next(l for l in range(6) if 20 * 4 ** l >= nf))
    f, rng = np.asarray(f)[:nf], np.random.default_rng(1)
    nv = len(v) + nv_extra
    if kind == "faces shuffled":
        f = f[rng.permutation(nf)]
    if kind == "vertices shuffled":
        f = rng.permutation(nv)[f]
    if kind == "corners apart":  # no face shares a vertex
        nv = max(nv, 3 * nf)
        f = np.arange(3 * nf).reshape(-1, 3)
    F = torch.tensor(f, dtype=torch.int32, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(nf)
    m = torch.rand((nf, nf, 3, 3), generator=g, dtype=torch.float32, device="cuda")
    ids = F.long()
    ref = torch.zeros(nv * nv, dtype=torch.float64, device="cuda")
    at = ids[:, None, :, None] * nv + ids[None, :, None, :]
    ref.index_add_(0, at.expand(nf, nf, 3, 3).reshape(-1), m.double().reshape(-1))
    got = pkg.utils.pack_matrix_tight(1, m, torch.zeros((nv, 3), device="cuda"), F).reshape(-1).double()
    assert (torch.linalg.norm(got - ref) / torch.linalg.norm(ref)).item() < TOL


def test_face_order(pkg):
    """The two figures the choice is made by, against their definition."""
    import ctypes

    v, f = pkg.meshes.icosphere(3)
    for g in (np.asarray(f), np.asarray(f)[np.random.default_rng(3).permutation(len(f))], np.asarray(f)[:21], np.asarray(f)[:1]):
        n = len(g)
        ids, sectors = [], []
        for s in range(16):
            a, b = max(n - 10, 0) * s // 15, max(n - 32, 0) * s // 15
            ids.append(len(set(g[a:a + 10].reshape(-1).tolist())))
            sectors.append(sum(len(set((g[b:b + 32, c] // 8).tolist())) for c in range(3)))
        order = (ctypes.c_int32 * 2)()
        F = torch.tensor(g, dtype=torch.int32, device="cuda")
        assert not pkg.utils.indices_outside(F, len(v), order)
        assert list(order) == [sum(ids) // 16, sum(sectors) // 16]
        F[0, 1] = len(v)
        assert pkg.utils.indices_outside(F, len(v), order)
        F[0, 1] = -1
        assert pkg.utils.indices_outside(F, len(v), order)
