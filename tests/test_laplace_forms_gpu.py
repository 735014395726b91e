"""The packed FP32 Laplace operators on both sides of the lines between their two kernels (a block per test face; groups
of test faces per block): mesh sizes, row windows, meshes whose consecutive faces share vertices and meshes whose do
not, sheets a hundredth of an edge apart.  Reference: the stored panels, packed in FP64.  Tolerance as in
test_vertex_slots_gpu.py."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 1e-6


def _rel(a, b):
    return (torch.linalg.norm(a.double() - b.double()) / torch.linalg.norm(b.double())).item()


def _mesh(pkg, nf, kind):
    v, f = pkg.meshes.icosphere(next(l for l in range(6) if 20 * 4 ** l >= nf))
    f = np.asarray(f)[:nf]
    used, inv = np.unique(f, return_inverse=True)
    v, f = np.asarray(v)[used], inv.reshape(-1, 3)
    if kind == "shuffled":
        f = f[np.random.default_rng(0).permutation(nf)]
    if kind == "sheets":
        h = nf // 2
        v, f = np.concatenate((v, 1.003 * v)), np.concatenate((f[:h], f[:nf - h] + v.shape[0]))
    return torch.tensor(v, dtype=torch.float32, device="cuda"), torch.tensor(f, dtype=torch.int32, device="cuda")


def _reference(pkg, v, f, op, near, rows):
    L = pkg.layers
    m = L.hypersingular_from_v0(v, f, L.laplace_sym_panels(v, f, 1, 0, near)) if op == 3 else \
        L.laplace_sym_panels(v, f, op, 1, near)
    m[:rows[0]] = 0
    m[rows[1]:] = 0
    return pkg.utils.pack_matrix_tight(1, m.double(), v.double(), f)


@pytest.mark.parametrize("kind", ["ordered", "shuffled", "sheets"])
@pytest.mark.parametrize("nf", [149, 150, 2601, 3599, 3600, 4799, 4800])
@pytest.mark.parametrize("op", [1, 2, 3])
def test_sizes(pkg, nf, kind, op):
    v, f = _mesh(pkg, nf, kind)
    near = pkg.layers.laplace_near_pairs(f, v.shape[0])
    ref = _reference(pkg, v, f, op, near, (0, nf))
    assert _rel(pkg.layers.laplace_sym_tight(v, f, op, near), ref) < TOL


@pytest.mark.parametrize("kind", ["ordered", "shuffled", "sheets"])
@pytest.mark.parametrize("nf,rows", [(120, (0, 120)), (150, (3, 66)), (150, (3, 67)), (640, (0, 1)), (640, (100, 117)),
                                     (640, (639, 640)), (640, (0, 63)), (640, (5, 69)), (640, (320, 640)),
                                     (3599, (7, 518)), (3600, (7, 518)), (4800, (7, 519))])
@pytest.mark.parametrize("op", [1, 2, 3])
def test_row_windows(pkg, nf, rows, kind, op):
    v, f = _mesh(pkg, nf, kind)
    near = pkg.layers.laplace_near_pairs(f, v.shape[0])
    ref = _reference(pkg, v, f, op, near, rows)
    got = pkg.layers.laplace_sym_tight(v, f, op, near, rows=rows)
    assert _rel(got, ref) < TOL
    assert _rel(pkg.layers.laplace_sym_tight(v, f, op, near, rows=rows, out=got.clone()), 2 * ref) < TOL  # accumulates
