"""fp32 at 32 bits in blocks of several warp rows (an instance of its own): block
sizes 1,024 to 4,096, ends inside a block and a tile, and blocks that hold NaNs,
infinities, subnormals or zeros only.  Bytes and values equal the oracle's."""
import numpy as np
import pytest
import torch

import frsz_b200
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E", [1024, 2048, 4096])
@pytest.mark.parametrize("n", [1, 4096, 4097, 3 * 4096, 50_003])
def test_equals_oracle(cuda, E, n):
    rng = np.random.default_rng(E + n)
    x = (rng.standard_normal(n) * 2.0 ** rng.integers(-40, 40, n)).astype(np.float32)
    for b, v in enumerate((np.nan, -np.inf, np.inf, 1e-42, 0.0)):
        sl = slice(2 * b * E, (2 * b + 1) * E)
        if v in (1e-42, 0.0):
            x[sl] = v
        elif x[sl].size:
            x[sl][rng.integers(x[sl].size)] = v
    buf = torch.full((frsz_b200.compressed_size(np.float32, 32, E, n) + 64,), 0xA5, dtype=torch.uint8, device="cuda")
    frsz_b200.compress(torch.from_numpy(x).cuda(), 32, E, out=buf[:-64])
    want = oracle.compress(x, 32, E, canary=0xA5)
    got = buf.cpu().numpy()
    assert np.array_equal(got[:-64], want) and (got[-64:] == 0xA5).all()
    y = frsz_b200.decompress(buf[:-64], n, torch.float32, 32, E).cpu().numpy()
    assert np.array_equal(y.view(np.uint8), oracle.decompress(want, n, np.float32, 32, E).view(np.uint8))
