"""One block per lane: block sizes that no lane-segment kernel takes, from 9 to
past 128 values, every word width and block-byte remainder, arrays that end
inside a block, a warp's 32 blocks and a 16-byte access, and blocks with NaNs,
infinities and tiny values.  Bytes (with canaries) and values equal the
oracle's."""
import numpy as np
import pytest
import torch

import frsz_b200
import oracle
from frsz_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("E", [9, 10, 13, 15, 17, 18, 22, 24, 28, 31, 40, 50, 63, 90, 100, 127, 129, 150, 201, 300])
def test_equals_oracle(cuda, dtype, E):
    f32 = dtype == np.float32
    tdt = torch.float32 if f32 else torch.float64
    lengths = (1, E - 1, E, 31 * E + 1, 32 * E, 32 * E + E // 2, 33 * E, 97 * E + 5)
    x = workloads.loguniform_np(max(lengths), dtype, E, lo=-6, hi=6)
    x[3 * E] = np.nan
    x[7 * E + 1] = -np.inf
    x[20 * E:21 * E] *= dtype(1e-37 if f32 else 1e-300)
    x[40 * E:41 * E] = 0
    for i, bits in enumerate(range(4, (32 if f32 else 64) + 1)):
        n = lengths[i % len(lengths)] if bits not in (8, 13, 16, 21, 32, 40) else lengths[-1]
        ref = oracle.compress(x[:n], bits, E, canary=0x5C)
        buf = torch.full((ref.size + 64,), 0x5C, dtype=torch.uint8, device="cuda")
        frsz_b200.compress(torch.from_numpy(x[:n].copy()).cuda(), bits, E, out=buf)
        got = buf.cpu().numpy()
        assert np.array_equal(got[:ref.size], ref), (bits, n)
        assert np.all(got[ref.size:] == 0x5C)
        want = oracle.decompress(ref, n, dtype, bits, E)
        out = torch.full((n + 32,), 5.0, dtype=tdt, device="cuda")
        frsz_b200.decompress(torch.from_numpy(ref).cuda(), n, dtype, bits, E, out=out)
        y = out.cpu().numpy()
        assert np.array_equal(y[:n].view(np.uint8), want.view(np.uint8)), (bits, n)
        assert np.all(y[n:] == 5.0)
