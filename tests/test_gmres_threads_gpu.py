"""Solves of different sizes at the same time, each in a host thread and a stream of its own: the limit on
a kernel's shared memory belongs to the process, so a small solve must not lower it under a large
one between two of its cycles.  Tolerance: the solver's own promise, checked in FP64."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _system(n, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    A = torch.randn((n, n), generator=g, dtype=dtype, device="cuda") * (0.3 / n ** 0.5)
    A += torch.eye(n, dtype=dtype, device="cuda")
    return A, torch.randn(n, generator=g, dtype=torch.complex128 if dtype.is_complex else torch.float64, device="cuda")


@pytest.mark.parametrize("dtype", [torch.complex64, torch.float64])
def test_large_and_small_solves_together(pkg, dtype):
    solve = pkg.mesh_MOM_3d.gmres if dtype.is_complex else pkg.mesh_MOM_3d.gmres_real
    systems = [_system(n, dtype, n) for n in (3000, 40, 41, 700)]
    torch.cuda.synchronize()
    errors, done = [], threading.Event()

    def run(A, b, times):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(times):
                    if done.is_set():
                        break
                    x, (info,) = solve(A, b, restart=4, tol=1e-9)  # several cycles each
                    r = (torch.linalg.norm(b - A.to(b.dtype) @ x) / torch.linalg.norm(b)).item()
                    if not info["converged"] or r > 1.01e-9:
                        errors.append((A.shape[0], info, r))
        except Exception as e:  # noqa: BLE001
            errors.append((A.shape[0], e))
        if A.shape[0] == 3000:
            done.set()

    threads = [threading.Thread(target=run, args=(*s, 30 if s[0].shape[0] == 3000 else 10 ** 6)) for s in systems]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not any(t.is_alive() for t in threads) and not errors, errors[:3]
