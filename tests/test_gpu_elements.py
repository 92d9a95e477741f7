"""Random access over word widths, odd block sizes and the last elements: the
block index comes from a shift or a multiply-high, so every index around block
boundaries is compared with the oracle's decode, bit for bit."""
import numpy as np
import pytest
import torch

import frsz_b200
import oracle


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("E", [1, 2, 3, 5, 32, 100, 1000, 65535, 65536])
def test_block_boundaries(cuda, dtype, E):
    rng = np.random.default_rng(E)
    n = 3 * E + 70_001
    x = rng.standard_normal(n).astype(dtype)
    edges = np.unique(np.clip(np.concatenate([np.arange(0, n, E) + d for d in (-1, 0, 1)]), 0, n - 1))
    idx = np.concatenate([rng.permutation(edges)[:20_000], [0, n - 1, n, n + 5, 2 ** 40]]).astype(np.int64)
    for bits in (4, 8, 9, 16, 17, 31, 32) + ((33, 51, 64) if dtype == np.float64 else ()):
        ref = oracle.compress(x, bits, E)
        want = oracle.decompress(ref, n, dtype, bits, E)
        out = torch.full((idx.size,), 77.0, dtype=torch.float32 if dtype == np.float32 else torch.float64, device="cuda")
        frsz_b200.decompress_elements(torch.from_numpy(ref).cuda(), n, dtype, bits, E, torch.from_numpy(idx).cuda(), out=out)
        got = out.cpu().numpy()
        assert np.array_equal(got[:-3].view(np.uint8), want[idx[:-3]].view(np.uint8)), bits
        assert np.all(got[-3:] == 77.0)  # indices past the array write nothing
