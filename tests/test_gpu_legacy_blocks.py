"""The legacy codec's kernels where they change behaviour: array ends inside
and at the end of a warp's 32 blocks, steps for which the decoder rounds its
sums by conversion instead of integer arithmetic, sums that end halfway
between floats, and blocks that mix values inside and outside the integer
quantizer's range.  Everything equals the oracle bit for bit."""
import numpy as np
import pytest
import torch

import oracle
from frsz_b200 import legacy

LENGTHS = (1, 255, 256, 257, 32 * 256 - 1, 32 * 256, 32 * 256 + 1, 33 * 256 + 77, 65 * 256)
# 2 eps at 2^-66, 2^-64 (the decoder's bound), dyadic steps (sums on ties), a decimal one, 2^96 and 2^98
EPSILONS = (2.0 ** -67, 2.0 ** -65, 2.0 ** -12, 0.25, 1e-3, 2.0 ** 95, 2.0 ** 97)


def _same(got, want):
    return np.array_equal(got.view(np.uint8), want.view(np.uint8))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", LENGTHS)
def test_equals_oracle(cuda, dtype, n):
    rng = np.random.default_rng(n)
    tdt = torch.float32 if dtype == np.float32 else torch.float64
    for eps in EPSILONS:
        step = 2.0 * eps
        # quantized values of a random walk, some halves, and a few beyond +-2^24 and Inf / NaN
        x = np.cumsum(rng.integers(-9000, 9001, n)) * 0.5
        x[rng.random(n) < 0.001] *= 2.0 ** 12
        with np.errstate(over="ignore"):
            x = (x * step).astype(dtype)
        if n > 300:
            x[n // 2], x[n // 3], x[n // 5] = np.inf, np.nan, -0.0
        want = oracle.frsz1_compress(x, eps)
        out = torch.full((n + 32,), 77, dtype=torch.int16, device="cuda")
        legacy.compress(torch.from_numpy(x).cuda(), eps, out=out[:n])
        assert np.array_equal(out.cpu().numpy()[:n], want), eps
        assert bool((out[n:] == 77).all())
        for q in (want, rng.integers(-32768, 32768, n).astype(np.int16), rng.integers(-3, 4, n).astype(np.int16)):
            t = torch.from_numpy(q).cuda()
            for own in (True, False):
                y = torch.full((n + 32,), -3.0, dtype=tdt, device="cuda")
                legacy.decompress(t, tdt, eps, own_deltas=own, out=y[:n])
                got = y.cpu().numpy()
                assert _same(got[:n], oracle.frsz1_decompress(q, dtype, eps, own_deltas=own)), (eps, own)
                assert np.all(got[n:] == -3.0)


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [4, 8])
def test_output_off_sixteen_bytes(cuda, shift):
    """fp64 values whose int16 stream starts 8 bytes (4 codes) off."""
    x = np.random.default_rng(shift).standard_normal(1000)
    out = torch.zeros(1000 + shift, dtype=torch.int16, device="cuda")
    legacy.compress(torch.from_numpy(x).cuda(), 1e-3, out=out[shift:])
    assert np.array_equal(out.cpu().numpy()[shift:], oracle.frsz1_compress(x, 1e-3))
