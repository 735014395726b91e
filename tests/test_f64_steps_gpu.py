"""The kernels' own FP64 reciprocal root, root, quotient, sine and cosine (csrc/f64_steps.cuh) against CUDA's, over normal
arguments of any size.

Bounds, in units of the last place u of CUDA's result, which is itself within 1 u (CUDA's documented bounds: rsqrt 1, sqrt
and division correctly rounded, sin and cos of the table and of torch 2): the reciprocal root's step rounds x y, t and the last sum, at most
1.5 u together, and the approximation's 2^-58.7 adds 0.02: 3 u apart. The root multiplies it by x, 0.5 u more: 3 u.
The quotient is corrected by its residual: 0.5 u and a little, 2 u apart. Sine and cosine are sums of numbers below 1 whose
parts round at 2^-54 to 2^-53 (table, products, last sum) and drop 8e-18: 3e-16 absolute, and the reference's
angle, exact in 256ths of a turn, rounds by 2^-53 of itself: 8e-16 for angles up to pi."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(pkg, which, x, y=None):
    out = torch.empty_like(x)
    L = pkg._lib
    L.call("mb_f64_steps", which, L.ptr(x), L.ptr(y), x.numel(), L.ptr(out), L.stream_of(x))
    return out


def _ulps(got, ref):
    a, b = got.cpu().numpy(), ref.cpu().numpy()
    return np.max(np.abs(a - b) / np.spacing(np.abs(b)))


def _wide(n, seed, lo=-300.0, hi=300.0):
    """Mantissas over a binade, exponents over the range, and the numbers next to powers of two."""
    rng = np.random.default_rng(seed)
    x = np.concatenate((rng.uniform(1.0, 4.0, n), 10.0 ** rng.uniform(lo, hi, n)))
    p = 2.0 ** np.arange(-900, 901)
    return np.concatenate((x, p, np.nextafter(p, 0), np.nextafter(p, np.inf)))


def test_roots(pkg):
    x = torch.tensor(_wide(1 << 20, 1), device="cuda")
    assert _ulps(_run(pkg, 0, x), torch.rsqrt(x)) <= 3
    assert _ulps(_run(pkg, 1, x), torch.sqrt(x)) <= 3
    zero = torch.zeros(1, dtype=torch.float64, device="cuda")
    assert _run(pkg, 1, zero).item() == 0.0


def test_quotient(pkg):
    x, y = _wide(1 << 20, 2, -140, 140), _wide(1 << 20, 3, -140, 140)[::-1].copy()
    x, y = x[(x > 1e-140) & (x < 1e140)], y[(y > 1e-140) & (y < 1e140)]
    n = min(len(x), len(y))
    x, y = torch.tensor(x[:n], device="cuda"), torch.tensor(y[:n] * np.where(np.arange(n) % 2, 1.0, -1.0), device="cuda")
    assert _ulps(_run(pkg, 2, x, y), x / y) <= 2


@pytest.mark.parametrize("turns", [1.0, 4096.0])
def test_sine_and_cosine(pkg, turns):
    """x y = m / 2^26 exactly, in 256ths of a turn, over [0, turns) turns and the middles between the table's angles."""
    rng = np.random.default_rng(4)
    m = np.concatenate((rng.integers(0, int(turns * 256) << 26, 1 << 20), (np.arange(512) << 25)))  # < 2^53
    z = m / 2.0 ** 26
    x, y = torch.tensor(z * 8.0, device="cuda"), torch.full((len(z),), 0.125, dtype=torch.float64, device="cuda")
    f = np.mod(z, 256.0)  # exact
    f = np.where(f > 128.0, f - 256.0, f)  # exact
    a = torch.tensor(f * (np.pi / 128.0), device="cuda")
    assert (_run(pkg, 3, x, y) - torch.sin(a)).abs().max().item() <= 8e-16
    assert (_run(pkg, 4, x, y) - torch.cos(a)).abs().max().item() <= 8e-16
