"""Decompress of blocks of 3, 5, 6, 7 and 12 values by warps of 32 blocks: every
width, lengths around a warp's group, a CTA's groups and a partial last block,
with special values in some blocks; values equal the oracle's bit for bit and
nothing past the array is written."""
import numpy as np
import pytest
import torch

import frsz_b200
import oracle
from frsz_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("E", [3, 5, 6, 7, 12])
def test_equals_oracle(cuda, dtype, E):
    f32 = dtype == np.float32
    lengths = [b * E + d for b, d in ((1, 0), (31, 1), (32, 0), (32, E - 1), (33, 1), (128, 0), (257, 2), (513, E - 1))]
    top = max(lengths)
    x = workloads.loguniform_np(top, dtype, E, lo=-6, hi=6)
    x[5 * E:6 * E] = np.inf
    x[40 * E + 1] = np.nan
    x[60 * E:61 * E] *= dtype(1e-37 if f32 else 1e-300)
    for bits in range(4, (32 if f32 else 64) + 1):
        n = lengths[bits % len(lengths)]
        for n in (n, lengths[(bits + 3) % len(lengths)]):
            ref = oracle.compress(x[:n], bits, E)
            want = oracle.decompress(ref, n, dtype, bits, E)
            out = torch.full((n + 64,), 5.0, dtype=torch.float32 if f32 else torch.float64, device="cuda")
            frsz_b200.decompress(torch.from_numpy(ref).cuda(), n, dtype, bits, E, out=out)
            got = out.cpu().numpy()
            assert np.array_equal(got[:n].view(np.uint8), want.view(np.uint8)), (bits, n)
            assert np.all(got[n:] == 5.0)
