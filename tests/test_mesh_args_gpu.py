"""Face areas and normals in one kernel against the tensor functions, and the index range check.

Tolerance: a component of e0 x e1 is a difference of two products, rounded in an order that the
compiler may fuse: 4 eps |e0| |e1| on twice the area, that over the area on the normal."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mom():
    import importlib

    return importlib.import_module("mesh-ferrofluid_gb300").mesh_MOM_3d


def _mesh(nf, dtype, seed=0):
    g = torch.Generator().manual_seed(seed)
    v = torch.rand((nf + 2, 3), generator=g, dtype=torch.float64)
    f = torch.stack([torch.randperm(nf + 2, generator=g)[:3] for _ in range(nf)]) if nf else torch.zeros((0, 3))
    return v.to("cuda", dtype), f.to("cuda", torch.int32)


@pytest.mark.parametrize("nf", [0, 1, 255, 256, 257, 1025])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_face_geometry(mom, nf, dtype):
    v, f = _mesh(nf, dtype)
    if nf > 2:
        f[1] = f[1, 0]  # no area
    a, n = mom.face_geometry(v, f)
    ra, rn = mom.compute_face_areas(v, f), mom.compute_face_normals(v, f)
    assert a.shape == ra.shape == (nf, 1) and n.shape == rn.shape == (nf, 3) and a.dtype == n.dtype == dtype
    p = v[f.long()]
    tol = 4 * torch.finfo(dtype).eps * ((p[:, 1] - p[:, 0]).norm(dim=-1) * (p[:, 2] - p[:, 1]).norm(dim=-1))[:, None]
    assert torch.all((a - ra).abs() <= tol)
    assert torch.all((n - rn).abs() <= (tol / ra).nan_to_num(0.0) + torch.finfo(dtype).eps)


def test_face_geometry_leaves_gradients_and_other_layouts_to_the_tensor_functions(mom):
    v, f = _mesh(40, torch.float64)
    ref = mom.face_geometry(v, f)
    w = v.clone().requires_grad_(True)
    a, n = mom.face_geometry(w, f)
    assert a.requires_grad and n.requires_grad
    wide = torch.cat((v, v), 1)[:, :3]
    for x, g in ((w, f), (wide, f), (v, f.long()), (v.cpu(), f.cpu())):
        for got, want in zip(mom.face_geometry(x, g), ref):
            assert torch.allclose(got.detach().cpu(), want.cpu(), rtol=1e-13, atol=0)
    with torch.autograd.forward_ad.dual_level():
        d = torch.autograd.forward_ad.make_dual(v, torch.ones_like(v))
        assert torch.autograd.forward_ad.unpack_dual(mom.face_geometry(d, f)[0]).tangent is not None


# one thread, one block and its neighbours, more than the 304 blocks of 256 threads take in one pass
@pytest.mark.parametrize("count", [1, 255, 1024, 1025, 304 * 256 * 3 + 5])
def test_index_range(mom, count):
    x = torch.randint(0, 50, (count,), dtype=torch.int32, device="cuda")
    assert not mom._indices_outside(x, 50)
    for i in {0, count // 2, count - 1}:
        for bad in (-1, 50, 2**31 - 1, -2**31):
            y = x.clone()
            y[i] = bad
            assert mom._indices_outside(y, 50)
    assert not mom._indices_outside(x[:0], 0)
