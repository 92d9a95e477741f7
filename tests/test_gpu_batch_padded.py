"""Batched plans whose classes hold padded blocks, none, or both: the per-tile
kernels have an instance with the padded blocks' code and one without.  Bytes
and values equal the oracle's in every mode."""
import numpy as np
import pytest
import torch

import frsz_b200
import oracle
from frsz_b200 import BatchArray, BatchPlan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks", [(8,), (64,), (8, 64, 16)])
@pytest.mark.parametrize("per_tile", [True, False])
def test_classes(cuda, blocks, per_tile):
    rng = np.random.default_rng(len(blocks))
    arrays, inputs = [], []
    for dtype in (np.float32, np.float64):
        for bits in (9, 13, 21, 31, 33, 51):
            if dtype == np.float32 and bits > 32:
                continue
            for E in blocks:
                for n in (1, 2047, 4097, 30_001):
                    x = rng.standard_normal(n).astype(dtype)
                    t = torch.from_numpy(x).cuda()
                    size = frsz_b200.compressed_size(dtype, bits, E, n)
                    buf = torch.full((size,), 0x77, dtype=torch.uint8, device="cuda")
                    arrays.append(BatchArray(values=t, compressed=buf, bits=bits, block_size=E,
                                             decompressed=torch.zeros_like(t)))
                    inputs.append((x, bits, E))
    plan = BatchPlan(arrays)
    for c in (True, False):
        plan.configure(c, ctas_per_sm=2, one_cta_per_tile=per_tile)
    plan.compress()
    plan.decompress()
    torch.cuda.synchronize()
    for a, (x, bits, E) in zip(arrays, inputs):
        ref = oracle.compress(x, bits, E, canary=0x77)
        assert np.array_equal(a.compressed.cpu().numpy(), ref), (x.dtype, bits, E, x.size)
        want = oracle.decompress(ref, x.size, x.dtype, bits, E)
        assert np.array_equal(a.decompressed.cpu().numpy().view(np.uint8), want.view(np.uint8))
