"""Bases with blocks of zeros (sparse first vectors): they decode to exact zeros
beside dense neighbours, tiny blocks and blocks of -0.0, they meet infinities in
w and in the coefficients as zeros do, and a dot of nothing else is exact."""
import pytest
import torch

from frsz_b200 import CompressedBasis

pytestmark = pytest.mark.gpu
TOL = 1e-12  # order of summation, as in test_gpu_krylov.py
E = 32


def _basis(bits, n, m, seed):
    """Vectors whose blocks are kept, zeroed, made tiny or -0.0 at random; one
    vector is zero, and one dense."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    basis = CompressedBasis(m, n, bits=bits, block_size=E)
    nb = (n + E - 1) // E
    for j in range(m):
        v = torch.randn(nb, E, generator=g, device="cuda", dtype=torch.float64)
        kind = torch.randint(0, 64, (nb,), generator=g, device="cuda")
        if j == 1:
            v.zero_()
        elif j != 2:
            v[kind < 30] = 0.0
            v[kind == 60] = -0.0
            v[kind == 61] *= 2.0 ** -1000  # exponent outside the direct range, codes that are not zero
        basis.append(v.reshape(-1)[:n].contiguous())
    return basis, g


@pytest.mark.parametrize("bits", [16, 21, 24, 32, 48, 64])
@pytest.mark.parametrize("n,m", [(31, 3), (5_000, 1), (20_011, 2), (300_007, 9), (1_300_001, 5)])
def test_dot_and_axpy(cuda, bits, n, m):
    basis, g = _basis(bits, n, m, bits + m)
    V = torch.stack([basis.get(j) for j in range(m)])
    w = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    h = basis.dot(w)
    assert torch.all((h - V @ w).abs() <= TOL * (V.abs() @ w.abs()) + 1e-300)
    c = torch.randn(m, generator=g, device="cuda", dtype=torch.float64)
    y = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    want, scale = y + c @ V, y.abs() + c.abs() @ V.abs()
    basis.axpy(c, y)
    assert torch.all((y - want).abs() <= TOL * scale)


@pytest.mark.parametrize("bits", [16, 21, 24, 32, 48, 64])
def test_zeros_are_exact(cuda, bits):
    """One block of 2^-950 and zeros elsewhere: 32 * 2^-950 and nothing more."""
    n = 100_000
    basis = CompressedBasis(3, n, bits=bits, block_size=E)
    for j in range(3):
        v = torch.zeros(n, device="cuda", dtype=torch.float64)
        v[E * (500 + j):E * (501 + j)] = 2.0 ** -950
        basis.append(v)
    h = basis.dot(torch.ones(n, device="cuda", dtype=torch.float64))
    assert h.tolist() == [2.0 ** -945] * 3
    y = torch.zeros(n, device="cuda", dtype=torch.float64)
    basis.axpy(torch.full((3,), 2.0, device="cuda", dtype=torch.float64), y)
    want = torch.zeros_like(y)
    want[E * 500:E * 503] = 2.0 ** -949
    assert torch.equal(y, want)


@pytest.mark.parametrize("bits", [16, 32, 48, 64])
def test_zero_times_infinity(cuda, bits):
    n = 4096
    basis = CompressedBasis(2, n, bits=bits, block_size=E)
    basis.append(torch.zeros(n, device="cuda", dtype=torch.float64))
    basis.append(torch.ones(n, device="cuda", dtype=torch.float64))
    w = torch.ones(n, device="cuda", dtype=torch.float64)
    w[100] = float("inf")
    h = basis.dot(w)
    assert torch.isnan(h[0]) and torch.isinf(h[1])
    y = torch.ones(n, device="cuda", dtype=torch.float64)
    basis.axpy(torch.tensor([float("inf"), 0.0], device="cuda", dtype=torch.float64), y)
    assert torch.isnan(y).all()
