"""Compress where the block maxima are taken with floating-point instructions:
NaNs of every kind (quiet, signalling patterns, negative, payloads), +-Inf,
the largest finite values (fp64 from 2^1017 up has a high word that reads as
a float NaN), subnormals and zeros, in every position of a lane, through every
kind of instance (blocks below a lane, of a lane, of several rows, whole-block
tiles, half lanes, values off the 32-byte layout).  Bytes equal the oracle's."""
import numpy as np
import pytest
import torch

import frsz_b200
import oracle

pytestmark = pytest.mark.gpu


def special_values(dtype, n, seed):
    rng = np.random.default_rng(seed)
    f32 = dtype == np.float32
    x = rng.standard_normal(n).astype(dtype)
    u = x.view(np.uint32 if f32 else np.uint64)
    top = 0x7F7FFFFF if f32 else 0x7FEFFFFFFFFFFFFF
    inf = 0x7F800000 if f32 else 0x7FF0000000000000
    sign = 0x80000000 if f32 else 0x8000000000000000
    # finite: the largest, and (fp64) around 2^1016 .. 2^1018 where the high word crosses 0x7F800000
    finite = [top, 1, 0, sign, sign | 1, 0x00800000 if f32 else 1 << 52]
    if not f32:
        finite += [0x7F7FFFFF00000000, 0x7F80000000000000, 0x7F80000000000001, 0x7F800001FFFFFFFF, sign | 0x7F9ABCDE12345678]
    others = [inf, sign | inf, inf | 1, sign | inf | 1, inf | (1 << (22 if f32 else 51)), (1 << (32 if f32 else 64)) - 1, sign - 1]
    # sparse, so most blocks keep the plain path and a few mix
    for vals, share in ((finite, 0.002), (others, 0.001)):
        at = np.flatnonzero(rng.random(n) < share)
        u[at] = np.array([vals[i % len(vals)] for i in range(at.size)], dtype=u.dtype)
    return x


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("bits", [4, 5, 12, 13, 16, 21, 24, 28, 32, 40, 51, 64])
def test_bytes_equal_oracle(cuda, dtype, bits):
    if dtype == np.float32 and bits > 32:
        pytest.skip("fp32 has up to 32 bits")
    for E in (2, 4, 8, 16, 32, 128, 256, 512, 1024, 20, 24, 100, 120):
        for off in (0, 1):
            n = 20_000 + 7 * E + off
            x = special_values(dtype, n, bits * 1000 + E)
            t = torch.empty(n + off, dtype=torch.float32 if dtype == np.float32 else torch.float64, device="cuda")
            t[off:] = torch.from_numpy(x).cuda()
            size = frsz_b200.compressed_size(dtype, bits, E, n)
            buf = torch.full((size,), 0xA5, dtype=torch.uint8, device="cuda")
            frsz_b200.compress(t[off:], bits, E, out=buf)
            assert np.array_equal(buf.cpu().numpy(), oracle.compress(x, bits, E, canary=0xA5)), (E, off)
