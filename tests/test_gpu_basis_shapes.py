"""The fused basis kernels where their launch rules change: one or two vectors
or more, groups that end inside a launch's four, blocks of 4 and of 8 values
and more, lengths around a lane, a warp step and a slice, and the axpy's
change from four to eight values per thread.  Against torch fp64 on the
decompressed vectors; the sums differ from torch's only in order, so
|got - want| <= 1e-12 * sum(|terms|) as in test_gpu_krylov.py."""
import pytest
import torch

from frsz_b200 import CompressedBasis

pytestmark = pytest.mark.gpu
TOL = 1e-12
CANARY = 0xA5


def _check(bits, E, n, m, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    basis = CompressedBasis(m, n, bits=bits, block_size=E)
    for j in range(m):
        v = torch.randn(n, generator=g, device="cuda", dtype=torch.float64) * 2.0 ** (9 * (j % 5) - 18)
        v[torch.rand(n, generator=g, device="cuda") < 0.05] = 0.0
        if j % 3 == 2 and n > 600:  # a block or two outside the direct decode's exponents
            v[512:600] *= 2.0 ** 1000 if j % 2 else 2.0 ** -1000
        basis.append(v)
    V = torch.stack([basis.get(j) for j in range(m)])
    w = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    # the call stays inside the workspace it asks for
    size = basis.workspace.numel()
    room = torch.full((size + 4096,), CANARY, dtype=torch.uint8, device="cuda")
    basis.workspace = room[:size]
    h = basis.dot(w)
    assert bool((room[size:] == CANARY).all())
    for j in range(m):
        t = V[j] * w
        assert abs((h[j] - t.sum()).item()) <= TOL * t.abs().sum().item() + 1e-300, (j, h[j].item(), t.sum().item())
    assert torch.equal(h, basis.dot(w))
    c = torch.randn(m, generator=g, device="cuda", dtype=torch.float64)
    y = torch.randn(n + 8, generator=g, device="cuda", dtype=torch.float64)
    want, scale = y[:n].clone(), y[:n].abs()
    tail = y[n:].clone()
    basis.axpy(c, y[:n])
    for j in range(m):
        want = want + c[j] * V[j]
        scale = scale + (c[j] * V[j]).abs()
    assert bool(((y[:n] - want).abs() <= TOL * scale).all())
    assert torch.equal(y[n:], tail)


@pytest.mark.parametrize("bits", [16, 21, 24, 32, 48, 64])
@pytest.mark.parametrize("E", [4, 8, 32, 1024])
def test_small(cuda, bits, E):
    if (E * bits) % (8 if bits <= 8 else 16 if bits <= 16 else 32 if bits <= 32 else 64):
        pytest.skip("padded blocks: no fused kernel")
    for n, m in ((1, 1), (7, 2), (9, 3), (255, 5), (257, 4), (777, 9), (3071, 2), (12_289, 6)):
        _check(bits, E, n, m, n + m)


@pytest.mark.parametrize("bits", [16, 21, 24, 32, 48, 64])
@pytest.mark.parametrize("n,m", [(1_212_415, 3), (1_212_417, 2), (4_000_003, 1), (70_001, 130)])
def test_large(cuda, bits, n, m):
    _check(bits, 32, n, m, m)
