"""Host-array calls run after the work that the caller's stream already holds:
a pinned input that a copy still has to fill, with every mix of pinned and
ordinary memory that leaves one side ordinary, on the default and a side
stream, for one slice and for many.  The input holds other valid data before
the copy lands, so a call that does not wait gives those bytes."""
import numpy as np
import pytest
import torch

import frsz_b200
import oracle

pytestmark = pytest.mark.gpu


def _pinned(a, pin):
    t = torch.from_numpy(a.copy())
    return t.pin_memory() if pin else t


def _after_pending_work(dst, src):
    """Fills dst (pinned) on the current stream, about 20 ms from now."""
    torch.cuda._sleep(40_000_000)
    dst.copy_(src, non_blocking=True)


@pytest.mark.parametrize("n", [1000, 100_000, 3_000_001])
@pytest.mark.parametrize("side", [False, True])
@pytest.mark.parametrize("dtype,bits,E", [(np.float64, 32, 32), (np.float32, 13, 5)])
def test_input_still_on_its_way(cuda, dtype, bits, E, n, side):
    rng = np.random.default_rng(n + bits)
    old, new = (rng.standard_normal(n).astype(dtype) for _ in range(2))
    stream = torch.cuda.Stream() if side else torch.cuda.current_stream()
    ref_old, ref = (oracle.compress(x, bits, E, canary=0x5A, threads=4) for x in (old, new))
    want = oracle.decompress(ref, n, dtype, bits, E, threads=4)
    new_dev, ref_dev = torch.from_numpy(new).cuda(), torch.from_numpy(ref).cuda()
    x, buf = _pinned(old, True), _pinned(ref_old, True)
    out, y = np.full(ref.size, 0x5A, dtype=np.uint8), np.zeros(n, dtype=dtype)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        _after_pending_work(x, new_dev)
        frsz_b200.compress_host(x.numpy(), bits, E, out=out)
        assert np.array_equal(out, ref)
        _after_pending_work(buf, ref_dev)
        frsz_b200.decompress_host(buf.numpy(), n, dtype, bits, E, out=y)
        assert np.array_equal(y.view(np.uint8), want.view(np.uint8))


@pytest.mark.parametrize("pin_in", [False, True])
@pytest.mark.parametrize("pin_out", [False, True])
@pytest.mark.parametrize("decompress", [False, True])
def test_mixed_memory(cuda, pin_in, pin_out, decompress):
    """Both directions, each side pinned or not; the caller's bytes that the
    format leaves alone stay."""
    dtype, bits, E, n = np.float64, 21, 7, 2_500_003
    x = np.random.default_rng(5).standard_normal(n)
    ref = oracle.compress(x, bits, E, canary=0x5A, threads=4)
    if decompress:
        out = _pinned(np.zeros(n), pin_out).numpy()
        frsz_b200.decompress_host(_pinned(ref, pin_in).numpy(), n, dtype, bits, E, out=out)
        want = oracle.decompress(ref, n, dtype, bits, E, threads=4)
        assert np.array_equal(out.view(np.uint8), want.view(np.uint8))
    else:
        out = _pinned(np.full(ref.size, 0x5A, dtype=np.uint8), pin_out).numpy()
        frsz_b200.compress_host(_pinned(x, pin_in).numpy(), bits, E, out=out)
        assert np.array_equal(out, ref)


def test_output_still_being_read(cuda):
    """A pinned output that a pending copy still reads keeps its bytes until then."""
    n, bits, E = 1_000_001, 32, 32
    x = np.random.default_rng(6).standard_normal(n)
    ref = oracle.compress(x, bits, E, canary=0x5A, threads=4)
    out = _pinned(np.full(ref.size, 0x5A, dtype=np.uint8), True)
    seen = torch.zeros(ref.size, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    torch.cuda._sleep(40_000_000)
    seen.copy_(out, non_blocking=True)
    frsz_b200.compress_host(x, bits, E, out=out.numpy())
    torch.cuda.synchronize()
    assert bool((seen == 0x5A).all())
    assert np.array_equal(out.numpy(), ref)
