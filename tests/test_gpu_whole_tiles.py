"""Kernels that take one tile per CTA, whole tiles apart from the partial last
one: lengths around whole tiles (of 4,096 fp32 / 2,048 fp64 values, half of that
for the narrower CTAs), through every kind of instance that does and does not
split or loop.  Bytes and values equal the oracle's, nothing past them is written."""
import numpy as np
import pytest
import torch

import frsz_b200
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,bits", [(np.float32, b) for b in (4, 6, 8, 12, 13, 15, 16, 19, 23, 28, 29, 32)]
                         + [(np.float64, b) for b in (4, 6, 8, 13, 16, 21, 23, 24, 33, 36, 40, 51, 64)])
def test_lengths_around_tiles(cuda, dtype, bits):
    tile = 4096 if dtype == np.float32 else 2048
    tt = torch.float32 if dtype == np.float32 else torch.float64
    for E in (1, 2, 4, 8, 32, 256, 512, 1024, 18, 20, 24, 96):
        for off in (0, 1):
            for n in (tile - 1, tile, tile + 1, 2 * tile, 3 * tile + 5, 4 * tile - tile // 2):
                x = np.random.default_rng(bits * 100 + E + n).standard_normal(n).astype(dtype)
                t = torch.empty(n + off, dtype=tt, device="cuda")
                t[off:] = torch.from_numpy(x).cuda()
                buf = torch.full((frsz_b200.compressed_size(dtype, bits, E, n) + 64,), 0xA5, dtype=torch.uint8, device="cuda")
                frsz_b200.compress(t[off:], bits, E, out=buf[:-64])
                want = oracle.compress(x, bits, E, canary=0xA5)
                got = buf.cpu().numpy()
                assert np.array_equal(got[:-64], want) and (got[-64:] == 0xA5).all(), (E, off, n)
                y = torch.full((n + off + 8,), 7.0, dtype=tt, device="cuda")
                frsz_b200.decompress(buf[:-64], n, tt, bits, E, out=y[off:off + n])
                out = y.cpu().numpy()
                assert np.array_equal(out[off:off + n].view(np.uint8), oracle.decompress(want, n, dtype, bits, E).view(np.uint8)), (E, off, n)
                assert (out[off + n:] == 7).all() and (out[:off] == 7).all(), (E, off, n)
