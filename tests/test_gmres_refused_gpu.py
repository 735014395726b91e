"""The solver where the driver refuses a cooperative launch, from the first cycle on or from a later one: it goes
on as launches.  The refusal comes from a stand-in for cudaLaunchCooperativeKernel, preloaded into a
process of its own.  Tolerance: the solver's own promise, checked in FP64."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

STAND_IN = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdlib.h>
typedef struct { unsigned x, y, z; } d3;
typedef int (*launch)(const void*, d3, d3, void**, size_t, void*);
static int calls;
int cooperative_calls(void) { return calls; }
int cudaLaunchCooperativeKernel(const void* f, d3 grid, d3 block, void** args, size_t bytes, void* stream) {
    if (++calls >= atoi(getenv("REFUSE_FROM"))) return atoi(getenv("REFUSE_WITH"));
    return ((launch)dlsym(RTLD_NEXT, "cudaLaunchCooperativeKernel"))(f, grid, block, args, bytes, stream);
}
"""
SOLVE = r"""
import ctypes, importlib, json, torch
pkg = importlib.import_module("mesh-ferrofluid_gb300")
out = []
for dt in (torch.complex64, torch.float32, torch.float64):
    g = torch.Generator(device="cuda").manual_seed(3)
    A = torch.randn((300, 300), generator=g, dtype=dt, device="cuda") * 0.02 + torch.eye(300, dtype=dt, device="cuda")
    b = torch.randn(300, generator=g, dtype=torch.complex128 if dt.is_complex else torch.float64, device="cuda")
    f = pkg.mesh_MOM_3d.gmres if dt.is_complex else pkg.mesh_MOM_3d.gmres_real
    try:
        x, (i,) = f(A, b, restart=3, tol=1e-9)
    except pkg._lib.MeshBEMError as e:
        out.append(str(e))
        continue
    out.append([i["converged"], i["iterations"], i["restarts"], (torch.linalg.norm(b - A.to(b.dtype) @ x) / torch.linalg.norm(b)).item()])
print(json.dumps([out, ctypes.CDLL(None).cooperative_calls()]))
"""


def _run(tmp_path, start, error):
    src, lib = tmp_path / "stand_in.c", tmp_path / "stand_in.so"
    src.write_text(STAND_IN)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", str(src), "-o", str(lib), "-ldl"], check=True)
    repo = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, LD_PRELOAD=str(lib), REFUSE_FROM=str(start), REFUSE_WITH=str(error))
    p = subprocess.run([sys.executable, "-c", SOLVE], cwd=repo, env=env, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]
    return json.loads(p.stdout.strip().splitlines()[-1])


def test_a_refused_launch_goes_on_as_launches(tmp_path):
    plain, calls = _run(tmp_path, 10 ** 6, 0)
    assert calls >= 9 and all(c and r <= 1.01e-9 for c, _, _, r in plain)
    for start in (1, 3):
        for error in (720, 801):  # too large for this context; not supported
            got, n = _run(tmp_path, start, error)
            assert n >= start
            for (c, it, cyc, r), (_, it0, cyc0, _) in zip(got, plain):
                assert c and r <= 1.01e-9
                assert abs(it - it0) <= 3 and abs(cyc - cyc0) <= 1  # a residual near the tolerance: one cycle more or less


def test_another_error_is_reported(tmp_path):
    got, _ = _run(tmp_path, 1, 1)
    assert all(isinstance(m, str) and "gmres cycle" in m for m in got)
