"""Host arrays through the staged path: lengths around one slice, two slice
sizes and many slices, blocks of one value (the largest compressed form) up to
65,536, arrays at odd addresses, pinned memory on one side, and calls from
several threads.  Bytes and values equal the oracle's; what the format leaves
unwritten keeps the caller's bytes."""
import threading

import numpy as np
import pytest
import torch

import frsz_b200
import oracle

pytestmark = pytest.mark.gpu
MIB = 1 << 20


def _round_trip(dtype, bits, E, n, seed, pin=None, off=0):
    x = np.empty(n + off, dtype=dtype)[off:]
    x[:] = np.random.default_rng(seed).standard_normal(n).astype(dtype)
    size = frsz_b200.compressed_size(dtype, bits, E, n)
    out = np.full(size, 0x5A, dtype=np.uint8)
    y = np.full(n, 9.0, dtype=dtype)
    if pin == "in":
        x = torch.from_numpy(x.copy()).pin_memory().numpy()
    elif pin == "out":
        out = torch.from_numpy(out).pin_memory().numpy()
        y = torch.from_numpy(y).pin_memory().numpy()
    frsz_b200.compress_host(x, bits, E, out=out)
    ref = oracle.compress(x, bits, E, canary=0x5A, threads=4)
    assert np.array_equal(out, ref), (dtype, bits, E, n)
    frsz_b200.decompress_host(out, n, dtype, bits, E, out=y)
    assert np.array_equal(y.view(np.uint8), oracle.decompress(ref, n, dtype, bits, E, threads=4).view(np.uint8))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("E", [1, 5, 32, 1000, 65536])
def test_slices(cuda, dtype, E):
    per = MIB // np.dtype(dtype).itemsize  # values of one slice
    for k, n in enumerate((1, per - 1, per, per + 1, per + 3 * E + 1, 8 * per, 8 * per + 1, 15 * per + 7)):
        _round_trip(dtype, (4, 13, 21, 32)[k % 4], E, n, n)
        if k in (3, 7):
            _round_trip(dtype, 32 if dtype == np.float32 else 64, E, n, n, pin=("in", "out")[k % 2], off=1)


def test_several_threads(cuda):
    errors = []

    def run(k):
        try:
            for i in range(3):
                _round_trip(np.float64, 32, 32, 300_001 + 70_000 * k + i, 10 * k + i)
        except BaseException as e:  # noqa: BLE001 - reported in the main thread
            errors.append(e)

    threads = [threading.Thread(target=run, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
