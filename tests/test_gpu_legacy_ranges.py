"""The legacy codec where its kernels choose: blocks whose largest magnitude lies
just inside or outside the integer quantizer's range, by values of either sign,
NaN, infinities and (fp64) values past 2^1017; pointers on and off the vector
layout; and a last block of every length modulo 8 and around the decoder's pieces
of 64 values.  Everything equals the oracle bit for bit."""
import numpy as np
import pytest
import torch

import oracle
from frsz_b200 import legacy

pytestmark = pytest.mark.gpu


def _off(a, off, fill):
    t = torch.full((a.size + off + 32,), fill, dtype=torch.from_numpy(a[:0]).dtype, device="cuda")
    t[off:off + a.size] = torch.from_numpy(a).cuda()
    return t, t[off:off + a.size]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("off_in,off_out", [(0, 0), (1, 0), (0, 1), (3, 5)])
def test_range_edges(cuda, dtype, off_in, off_out):
    eps = 0.5  # p = x: values are their own quantized values
    top = 2.0 ** 24
    edges = [top - 1, top - 0.5, top, np.nextafter(dtype(top), dtype(0)), np.nextafter(dtype(top), dtype(np.inf)), top + 2,
             2.0 ** 30, 2.0 ** 31, 2.0 ** 40, np.inf, np.nan, float(np.finfo(dtype).max), 0.5, 0.0]
    if dtype == np.float64:
        edges += [2.0 ** 1017, 2.0 ** 1017 * (1 + 2.0 ** -30), np.nextafter(0.5, 0.0), 5e-324]
    rng = np.random.default_rng(off_in + off_out)
    x = (rng.integers(-40000, 40001, 256 * len(edges) * 2 + 100) * 0.5).astype(dtype)
    for k, e in enumerate(edges * 2):
        x[256 * k + int(rng.integers(256))] = e if k < len(edges) else -e
    want = oracle.frsz1_compress(x, eps)
    _, xv = _off(x, off_in, 9.0)
    whole, out = _off(np.full(x.size, 77, dtype=np.int16), off_out, 77)
    legacy.compress(xv, eps, out=out)
    assert np.array_equal(out.cpu().numpy(), want)
    assert bool((whole[off_out + x.size:] == 77).all()) and bool((whole[:off_out] == 77).all())


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("blocks", [0, 1, 3, 31, 32])
def test_last_block(cuda, dtype, blocks):
    tdt = torch.float32 if dtype == np.float32 else torch.float64
    rng = np.random.default_rng(blocks)
    for tail in (0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 63, 64, 65, 127, 128, 129, 191, 200, 255):
        n = 256 * blocks + tail
        if n == 0:
            continue
        q = rng.integers(-32768, 32768, n).astype(np.int16)
        for eps, own in ((1e-3, True), (1e-3, False), (2.0 ** -70, True)):
            y = torch.full((n + 32,), -3.0, dtype=tdt, device="cuda")
            legacy.decompress(torch.from_numpy(q).cuda(), tdt, eps, own_deltas=own, out=y[:n])
            got = y.cpu().numpy()
            want = oracle.frsz1_decompress(q, dtype, eps, own_deltas=own)
            assert np.array_equal(got[:n].view(np.uint8), want.view(np.uint8)), (n, eps, own)
            assert np.all(got[n:] == -3.0)
        x = (np.cumsum(rng.integers(-900, 901, n)) * 2e-3).astype(dtype)
        out = torch.full((n + 32,), 77, dtype=torch.int16, device="cuda")
        legacy.compress(torch.from_numpy(x).cuda(), 1e-3, out=out[:n])
        assert np.array_equal(out.cpu().numpy()[:n], oracle.frsz1_compress(x, 1e-3)), n
        assert bool((out[n:] == 77).all())
