"""The preconditioner's columns at the sizes where its elimination changes path, and the preconditioned solver's
groups of eight steps at restart lengths around them.

Tolerance: the least-squares solution in FP32 is off by about the condition of the block (a few hundred here)
times 6e-8 times the columns' root: 2e-3, as for the sphere's columns.  Solver: its own tol of 1e-9, times the
system's condition (below 1e3)."""
import numpy as np
import pytest
import spai_reference as SR
import torch
from conftest import rel_err

pytestmark = pytest.mark.gpu


def _fan(n):
    t = 2 * np.pi * np.arange(n) / n
    v = np.concatenate(([[0, 0, 0.4]], np.stack((np.cos(t), np.sin(t), 0.1 * np.cos(3 * t)), 1)))
    return v, np.array([[0, 1 + i, 1 + (i + 1) % n] for i in range(n)])


def _strip(n):
    v = np.array([[i // 2, (i % 2) * 0.8, 0.2 * np.sin(i)] for i in range(n + 2)], float)
    return v, np.array([[i, i + 1, i + 2] if i % 2 == 0 else [i, i + 2, i + 1] for i in range(n)])


# (columns, rows) of a block: 3 x 3, 5 x 5, up to 9 x 13 in a strip, 16 x 16 (one group of four warps and columns),
# 18 x 18, 30 x 30 (one row of lanes), 32 x 32, 46 x 46
MESHES = {"face": lambda p: _strip(1), "two": lambda p: _strip(2), "strip": lambda p: _strip(12), "fan8": lambda p: _fan(8),
          "fan9": lambda p: _fan(9), "ico0": lambda p: p.meshes.icosphere(0), "fan16": lambda p: _fan(16),
          "fan23": lambda p: _fan(23)}


@pytest.mark.parametrize("mesh", list(MESHES))
def test_columns_of_small_and_full_blocks(pkg, cuda, mesh):
    v_np, f_np = MESHES[mesh](pkg)
    v = torch.tensor(np.asarray(v_np), dtype=torch.float32, device=cuda)
    f = torch.tensor(np.asarray(f_np), dtype=torch.int32, device=cuda)
    edges, fei, _ = pkg.utils.get_edge_unique(v, f)
    ne = edges.shape[0]
    Z = pkg.mesh_MOM_3d.assemble_Z_rwg_sym(v, f, fei, ne, 1.0)
    P = pkg.mesh_MOM_3d.spai_preconditioner(Z, v, f, fei, ne)
    assert P.status == 0
    cols, vals = P.cols.cpu().numpy(), P.vals.cpu().numpy()
    pats = SR.patterns(f.cpu().numpy(), fei.cpu().numpy(), ne)
    ref = SR.dense_m(SR.spai_columns(Z.cpu().numpy(), pats), ne)
    got = np.zeros((ne, ne), np.complex128)
    for i in range(ne):
        k = int((cols[i] >= 0).sum())
        assert np.array_equal(np.sort(cols[i, :k]), pats[i][0])
        got[i, cols[i, :k]] = vals[i, :k]
    assert rel_err(got, ref) < 2e-3


@pytest.mark.parametrize("restart", [1, 7, 8, 9, 16, 50])
@pytest.mark.parametrize("use_graph", [True, False])
def test_restart_lengths_around_the_groups(pkg, cuda, restart, use_graph):
    M = pkg.mesh_MOM_3d
    g = torch.Generator().manual_seed(restart)
    n = 200
    Z = torch.eye(n) + 0.35 * torch.randn(n, n, dtype=torch.complex64, generator=g) / n**0.5
    b = torch.randn(n, dtype=torch.complex128, generator=g)
    x, info = M.pgmres(Z.to(cuda), b.to(cuda), restart=restart, tol=1e-9, max_iters=400, use_graph=use_graph)
    assert info[0]["converged"] and info[0]["iterations"] <= 60
    assert rel_err(x.cpu().numpy(), torch.linalg.solve(Z.to(torch.complex128), b).numpy()) < 1e-6
