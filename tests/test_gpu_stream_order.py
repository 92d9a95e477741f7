"""Kernels that are launched before their predecessors end keep the stream's
order: long chains of library calls and torch work on the same buffers, with
nothing waited for in between, on the default and a side stream, across streams
by events, and captured into a graph with copies, fills and kernels between.
Each link's result is checked on the device at the end."""
import numpy as np
import pytest
import torch

import frsz_b200
from frsz_b200 import CompressedBasis, codec, legacy

pytestmark = pytest.mark.gpu

# (dtype, bits, E, n): one CTA, a few, a full wave and more; different kernels
SHAPES = [(torch.float64, 32, 32, 1000), (torch.float32, 16, 32, 70_001), (torch.float64, 21, 5, 30_011),
          (torch.float32, 8, 63, 50_003), (torch.float64, 13, 1024, 3_000_001), (torch.float32, 6, 128, 8_000_003),
          (torch.float64, 33, 1500, 100_003)]


def _links(shape, count, seed):
    """`count` inputs and what each decodes to, from separate, waited-for calls."""
    dtype, bits, E, n = shape
    g = torch.Generator(device="cuda").manual_seed(seed)
    xs = [torch.randn(n, generator=g, device="cuda", dtype=dtype) for _ in range(count)]
    want = []
    for x in xs:
        buf = codec.compress(x, bits, E)
        torch.cuda.synchronize()
        want.append(codec.decompress(buf, n, dtype, bits, E))
        torch.cuda.synchronize()
    return xs, want


def _chain(shape, xs, rounds, results):
    """Each link overwrites the input, the buffer and the output of the one before."""
    dtype, bits, E, n = shape
    x, y = torch.empty_like(xs[0]), torch.empty_like(xs[0])
    buf = torch.zeros(codec.compressed_size(dtype, bits, E, n), dtype=torch.uint8, device="cuda")
    for r in range(rounds):
        k = r % len(xs)
        if r % 3 == 0:
            x.copy_(xs[k])              # a copy before the compress
        elif r % 3 == 1:
            torch.mul(xs[k], 1.0, out=x)  # a kernel
        else:
            x.zero_()                   # a fill, then a kernel
            x.add_(xs[k])
        codec.compress(x, bits, E, out=buf)
        x.fill_(7.0)                    # must not reach the compress
        codec.decompress(buf, n, dtype, bits, E, out=y)
        buf.fill_(0x3C)                 # nor this the decompress
        results[r].copy_(y)
        y.zero_()


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("side", [False, True])
def test_chain(cuda, shape, side):
    xs, want = _links(shape, 3, 1)
    rounds = 24
    results = [torch.empty_like(want[0]) for _ in range(rounds)]
    torch.cuda.synchronize()
    if side:
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            _chain(shape, xs, rounds, results)
        s.synchronize()
    else:
        _chain(shape, xs, rounds, results)
    torch.cuda.synchronize()
    assert all(torch.equal(results[r], want[r % 3]) for r in range(rounds))


@pytest.mark.parametrize("shape", SHAPES[:5])
def test_captured_chain(cuda, shape):
    xs, want = _links(shape, 3, 2)
    results = [torch.empty_like(want[0]) for _ in range(9)]
    s = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):
        _chain(shape, xs, 3, results)
        s.synchronize()
        with torch.cuda.graph(g, stream=s):
            _chain(shape, xs, 9, results)
        for _ in range(3):
            for t in results:
                t.zero_()
            g.replay()
        s.synchronize()
    assert all(torch.equal(results[r], want[r % 3]) for r in range(9))


def test_across_streams(cuda):
    """Compress on one stream, decompress on the other, the buffer handed over by
    events both ways."""
    shape = SHAPES[4]
    dtype, bits, E, n = shape
    xs, want = _links(shape, 3, 3)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    buf = torch.zeros(codec.compressed_size(dtype, bits, E, n), dtype=torch.uint8, device="cuda")
    out = [torch.empty_like(want[0]) for _ in range(12)]
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    for r in range(12):
        with torch.cuda.stream(a):
            if r:
                a.wait_event(done)
            codec.compress(xs[r % 3], bits, E, out=buf)
            ready = torch.cuda.Event()
            ready.record(a)
        with torch.cuda.stream(b):
            b.wait_event(ready)
            codec.decompress(buf, n, dtype, bits, E, out=out[r])
            done = torch.cuda.Event()
            done.record(b)
    torch.cuda.synchronize()
    assert all(torch.equal(out[r], want[r % 3]) for r in range(12))


def test_solver_chain(cuda):
    """dot, axpy, element reads and the legacy codec in one chain, against the
    same calls waited for one by one."""
    n, m = 200_003, 7
    g = torch.Generator(device="cuda").manual_seed(4)
    basis = CompressedBasis(m, n, bits=16, block_size=32)
    vs = [torch.randn(n, generator=g, device="cuda", dtype=torch.float64) for _ in range(m)]
    w0 = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    idx = torch.randint(0, n, (5000,), generator=g, device="cuda")

    def steps(wait):
        w, got = w0.clone(), []
        basis.size = 0
        for j in range(m):
            basis.append(vs[j])
            wait()
            h = basis.dot(w)
            wait()
            basis.axpy(-1e-3 * h, w)
            wait()
            e = codec.decompress_elements(basis.buffers[j], n, torch.float64, 16, 32, idx)
            wait()
            q = legacy.compress(w, 1e-3)
            wait()
            got += [h, e, w.clone(), legacy.decompress(q, torch.float64, 1e-3, own_deltas=True)]
            wait()
        torch.cuda.synchronize()
        return got

    want = steps(torch.cuda.synchronize)
    for _ in range(3):
        assert all(torch.equal(a, b) for a, b in zip(steps(lambda: None), want))
    assert np.isfinite(want[-1].cpu().numpy()).all()
