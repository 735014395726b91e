"""The EFIE's separated pairs evaluated once per unordered pair against the row-by-row kernel
(``faces_range``), which evaluates every ordered pair, and against float64.

Tolerances: the two FP32 forms share the close and singular pairs, most of the norm, and each is
within some 1e-7 of the float64 matrix on the others, so they agree to 1e-6; against float64 the
pair form may not be further off than the rows (a tenth for the order of the additions)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 1e-6


def _rel(a, b):
    return (torch.linalg.norm(a.to(torch.complex128) - b.to(torch.complex128)) / torch.linalg.norm(b)).item()


def _mesh(pkg, kind):
    v, f = pkg.meshes.icosphere(0 if kind == "tiny" else 2)
    if kind == "shuffled":  # no shared edge within a group of 8 faces: more edges than places
        f = f[np.random.default_rng(0).permutation(f.shape[0])]
    if kind == "cut":  # 261 faces: partial groups of 8 and tiles of 128, boundary edges
        f = f[:261]
    if kind == "two":  # two spheres of unlike size
        g, h = pkg.meshes.icosphere(1)
        v, f = np.concatenate((v, 0.2 * g + [3.0, 0.1, 0.0])), np.concatenate((f, h + v.shape[0]))
    return v, f


@pytest.mark.parametrize("kind", ["tiny", "sphere", "shuffled", "cut", "two"])
@pytest.mark.parametrize("k", [0.4, 1.5, 20.0])  # all pairs far enough in phase; some; none
def test_pairs_equal_rows_and_float64(pkg, kind, k):
    ops, L = pkg.mesh_MOM_3d, pkg._lib
    v, f = _mesh(pkg, kind)
    v64, f = torch.tensor(v, device="cuda").float().double(), torch.tensor(f, dtype=torch.int32, device="cuda")
    v = v64.float()
    edges, fei, _ = pkg.utils.get_edge_unique(v, f)
    n = edges.shape[0]
    Z = ops.assemble_Z_rwg_sym(v, f, fei, n, k)
    rows = ops.assemble_Z_rwg_sym(v, f, fei, n, k, faces_range=(0, f.shape[0]))
    pairs = ops.near_pairs(f)
    L.call("mb_mom_sym_near_c64", L.ptr(v), v.shape[0], L.ptr(f), f.shape[0], L.ptr(fei), n, L.ptr(pairs), pairs.shape[0],
           float(k), L.ptr(rows), L.stream_of(v))
    assert _rel(Z, rows) < TOL
    ref = ops.assemble_Z_rwg_sym(v64, f, fei, n, k)
    assert _rel(Z, ref) <= 1.1 * _rel(rows, ref)
    again = ops.assemble_Z_rwg_sym(v, f, fei, n, k, out=Z.clone())  # accumulates
    assert _rel(again, 2 * Z) < TOL


# a part of a 32 x 32 tile, one tile, an even and an odd number of tile rows, a partial last one
@pytest.mark.parametrize("n_faces", [0, 1, 10, 20, 21, 42, 64, 107])
def test_fresh_matrix_equals_one_added_to_zeros(pkg, n_faces):
    """A matrix that is not passed in is summed above the diagonal and mirrored; one that is passed in is added to
    on both sides: the same additions in another order (a few 6e-8 of an entry's terms)."""
    ops = pkg.mesh_MOM_3d
    v, f = pkg.meshes.icosphere(2)
    v = torch.tensor(v, dtype=torch.float32, device="cuda")
    f = torch.tensor(f[:n_faces], dtype=torch.int32, device="cuda").reshape(-1, 3)
    fei = pkg.utils.get_edge_unique(v, f)[1] if n_faces else torch.zeros((0, 3), dtype=torch.int32, device="cuda")
    n = int(fei.max()) + 1 if n_faces else 5
    if n_faces == 107:  # edges that far faces share: terms on the diagonal
        fei = fei % (n - 40)
        n -= 40
    torch.full((n, n), float("nan"), device="cuda", dtype=torch.complex64)  # what the allocator may hand out
    Z = ops.assemble_Z_rwg_sym(v, f, fei, n, 0.4)
    ref = ops.assemble_Z_rwg_sym(v, f, fei, n, 0.4, out=torch.zeros((n, n), dtype=torch.complex64, device="cuda"))
    assert torch.linalg.norm(Z - ref) <= 5e-7 * torch.linalg.norm(ref)
