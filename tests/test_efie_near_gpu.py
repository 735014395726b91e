"""The complex64 entries of face pairs that share a vertex (closed form from the edges' common values) against the
complex128 ones (the general closed form, edge by edge).

Tolerance: each contribution is rounded to FP32 and up to four are added in FP32 (6e-8 each), the smooth part of
the kernel is FP32 with the hardware's sine (5e-7 of it, and it is k h of the entry): 1e-6 of the matrix."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pkg():
    import importlib

    return importlib.import_module("mesh-ferrofluid_gb300")


def _grid(n, z):
    x, y = np.meshgrid(np.arange(n + 1.0), np.arange(n + 1.0), indexing="ij")
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    p = (i * (n + 1) + j).reshape(-1)
    f = np.concatenate((np.stack((p, p + n + 1, p + n + 2), 1), np.stack((p, p + n + 2, p + 1), 1)))
    return np.stack((x, y, z(x, y)), -1).reshape(-1, 3), f


MESHES = {
    "one face": lambda pkg: (np.array([[0, 0, 0], [1, 0, 0], [0.2, 0.9, 0.1]]), np.array([[0, 1, 2]])),
    "flat": lambda pkg: _grid(4, lambda x, y: 0 * x),  # collinear edges, points in the planes of other faces
    "folded": lambda pkg: _grid(4, lambda x, y: 0.02 * np.abs(x - 2.0) + 3.0 * np.abs(y - 2.0)),
    "slivers": lambda pkg: (_grid(3, lambda x, y: 0.3 * np.sin(x * y))[0] * [1.0, 0.04, 1.0],
                            _grid(3, lambda x, y: x)[1]),
    "closed": lambda pkg: pkg.meshes.icosphere(1),
}


@pytest.mark.parametrize("mesh", list(MESHES))
@pytest.mark.parametrize("k", [0.05, 1.3])
@pytest.mark.parametrize("shift", [0.0, 3.0])
def test_near_pairs_complex64(pkg, mesh, k, shift):
    v, f = MESHES[mesh](pkg)
    v32 = torch.tensor(np.asarray(v) + shift, dtype=torch.float32, device="cuda")
    faces = torch.tensor(np.asarray(f), dtype=torch.int32, device="cuda")
    edges, fei, _ = pkg.utils.get_edge_unique(v32, faces)
    n = edges.shape[0]
    pairs = pkg.mesh_MOM_3d.near_pairs(faces)
    out = []
    for v, dt, sfx in ((v32, torch.complex64, "c64"), (v32.double(), torch.complex128, "c128")):
        z = torch.zeros((n, n), dtype=dt, device="cuda")
        pkg._lib.call(f"mb_mom_sym_near_{sfx}", pkg._lib.ptr(v), v.shape[0], pkg._lib.ptr(faces), faces.shape[0],
                      pkg._lib.ptr(fei), n, pkg._lib.ptr(pairs), pairs.shape[0], k, pkg._lib.ptr(z),
                      pkg._lib.stream_of(z))
        out.append(z.to(torch.complex128))
    assert torch.linalg.norm(out[1]) > 0
    assert torch.linalg.norm(out[0] - out[1]) <= 1e-6 * torch.linalg.norm(out[1])
