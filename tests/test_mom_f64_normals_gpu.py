"""The FP64 reference-rule entries with normals that are not perpendicular to their faces.

Face normals are an argument: smoothed vertex normals, or an STL file's that went through
float32, lean against their faces, and the entry's x.n then changes from test point to test
point.  Tolerance as in test_mom_f64_gpu.py, 3e-14 (1 + k R_max); leaving n.(x - A0) out changes
the matrix by 1e-3 at a tilt of 0.1, 4e-10 after float32."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tilt", [0.1, 1e-3, "float32"])
@pytest.mark.parametrize("gq", [2, 3, 4, 5])
def test_f64_entries_with_given_normals(oracle, tilt, gq):
    pkg = importlib.import_module("mesh-ferrofluid_gb300")
    u, k = pkg.utils, 2.0
    v_np, f_np = pkg.meshes.icosphere(1)
    v_np, f_np = np.asarray(v_np, np.float64) * np.array([1.0, 0.7, 0.4]), np.asarray(f_np, np.int32)
    v, f = torch.tensor(v_np, device="cuda"), torch.tensor(f_np, device="cuda")
    a, n = u.compute_face_areas(v, f).contiguous(), u.compute_face_normals(v, f).contiguous()
    if tilt == "float32":
        n = n.float().double()
    else:
        g = torch.Generator(device="cuda").manual_seed(5)
        n = torch.nn.functional.normalize(n + tilt * torch.randn(n.shape, generator=g, dtype=n.dtype, device="cuda"),
                                          dim=-1).contiguous()
    rules = [*u.get_gaussion_integration_points_and_weights(gq, device="cuda", dtype=torch.float64),
             *u.get_gaussion_integration_points_and_weights(gq - 1, device="cuda", dtype=torch.float64)]
    h = lambda t: t.cpu().numpy()  # noqa: E731
    ref = oracle.mom_zmat_fe(v_np, f_np, h(a), h(n), *(h(t) for t in rules), k)
    tol = 3e-14 * (1 + k * 2 * np.abs(v_np).max())
    ncol = 3 * f_np.shape[0]
    fei = torch.arange(ncol, dtype=torch.int32, device="cuda").reshape(-1, 3)
    z = pkg.mesh_MOM_3d.assemble_Z_rwg(v, f, a, n, fei, ncol, *rules, k)
    assert np.linalg.norm(h(z) - ref) <= tol * np.linalg.norm(ref)
    zr, zi = (torch.empty((1, ncol, ncol), dtype=torch.float64, device="cuda") for _ in range(2))
    pkg.mesh_MOM_3d.create_MOM_Zmat_3d_forward(v, f, a, n, *rules, zr, zi, k)
    assert np.linalg.norm(h(torch.complex(zr, zi))[0] - ref) <= tol * np.linalg.norm(ref)
