"""Packing by distinct test vertices (packed FP32 Laplace operators and stored panels) where its
cases change: more distinct vertices than places, partial blocks and groups, close separated faces.

Tolerances: both sides sum the same FP32 terms (relative rounding 6e-8 each, in another order, up
to 36 per entry): 1e-6 relative Frobenius, against FP64 1e-6 as well (the operators' FP32 error is
2e-7 on these meshes)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 1e-6


def _rel(a, b):
    return (torch.linalg.norm(a.double() - b.double()) / torch.linalg.norm(b.double())).item()


def _mesh(pkg, kind):
    v, f = pkg.meshes.icosphere(2 if kind != "fan" else 1)
    if kind == "shuffled":  # consecutive faces share nothing: 48 distinct vertices in 16 faces
        f = f[np.random.default_rng(0).permutation(f.shape[0])]
    if kind == "cut":  # 301 faces: partial blocks of 128 and groups of 16
        f = f[:301]
    if kind == "sheets":  # two patches a hundredth of an edge apart, no shared vertex
        v, f = np.concatenate((v, 1.003 * v)), np.concatenate((f, f + v.shape[0]))
    return torch.tensor(v, dtype=torch.float64, device="cuda"), torch.tensor(f, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("kind", ["sphere", "shuffled", "cut", "sheets"])
@pytest.mark.parametrize("op", [1, 2, 3])
def test_packed_operators(pkg, kind, op):
    L = pkg.layers
    v64, f = _mesh(pkg, kind)
    v = v64.float()
    near = L.laplace_near_pairs(f, v.shape[0])
    got = L.laplace_sym_tight(v, f, op, near)
    if op == 3:
        ref = L.hypersingular_tight(v, f, L.laplace_sym_panels(v, f, 1, 0, near))
    else:
        ref = pkg.utils.pack_matrix_tight(1, L.laplace_sym_panels(v, f, op, 1, near).double(), v, f)
    assert _rel(got, ref) < TOL
    if kind != "sheets":  # its separated pairs are as near as singular ones: FP32 differs by the rule's steepness
        assert _rel(got, L.laplace_sym_tight(v.double(), f, op, near)) < TOL
    k = f.shape[0] // 3 + 1  # row windows add up
    part = L.laplace_sym_tight(v, f, op, near, rows=(0, k))
    L.laplace_sym_tight(v, f, op, near, rows=(k, f.shape[0]), out=part)
    assert _rel(part, got) < TOL


@pytest.mark.parametrize("kind", ["sphere", "shuffled", "cut"])
def test_packed_panels(pkg, kind):
    v, f = _mesh(pkg, kind)
    nf, nv = f.shape[0], v.shape[0]
    g = torch.Generator(device="cuda").manual_seed(1)
    m = torch.rand((nf, nf, 3, 3), generator=g, dtype=torch.float32, device="cuda")
    ref = torch.zeros(nv * nv, dtype=torch.float64, device="cuda")
    ids = f.long()
    at = ids[:, None, :, None] * nv + ids[None, :, None, :]
    ref.index_add_(0, at.expand(nf, nf, 3, 3).reshape(-1), m.double().reshape(-1))
    assert _rel(pkg.utils.pack_matrix_tight(1, m, v.float(), f), ref.view(nv, nv)) < TOL
    odd = torch.empty(m.numel() + 1, dtype=torch.float32, device="cuda")[1:].view_as(m)  # 4-byte aligned panels
    odd.copy_(m)
    assert _rel(pkg.utils.pack_matrix_tight(1, odd, v.float(), f), ref.view(nv, nv)) < TOL
