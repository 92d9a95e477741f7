"""One block per lane at the lengths from which the dispatch takes it (short arrays
of long blocks go to other kernels): values read one by one and 16 bytes at a time,
images written by bytes, half-words and words, rows set apart on either side, and
blocks of up to 300 values.  Each case names the kernel family it is for, which is
read from a captured graph of the call, so a case that no longer reaches it fails.
Bytes (with canaries) and values equal the oracle's."""
import re

import numpy as np
import pytest
import torch

import frsz_b200
import oracle

pytestmark = pytest.mark.gpu

# block size, widths that both directions take one block per lane, widths of compress only
CASES = {
    np.float32: [(20, (5, 19, 27), ()), (22, (9,), ()), (24, (), (9, 21)), (28, (9, 27), ()), (31, (13, 24), ()),
                 (40, (), (13, 19)), (50, (5,), ()), (63, (4, 8, 24), ()), (90, (16,), ()), (100, (9, 13), ()),
                 (127, (6, 13), (32,)), (129, (4, 21), ()), (150, (8, 16), ()), (200, (5,), (21,)), (201, (13, 24), ()),
                 (300, (5,), ())],
    np.float64: [(20, (), (51,)), (22, (13,), ()), (28, (), (9, 27)), (31, (24,), (40, 64)), (50, (5, 9, 24), ()),
                 (63, (4, 13), (51,)), (90, (9, 13), ()), (100, (5,), ()), (129, (6, 27), ()), (150, (5, 8), ())],
}


def _kernels(call):
    """Names of the kernels a call launches."""
    driver = pytest.importorskip("cuda.bindings.driver")
    call()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        call()
    err, nodes, count = driver.cuGraphGetNodes(driver.CUgraph(g.raw_cuda_graph()), 16)
    assert int(err) == 0
    names = []
    for node in nodes[:count]:
        err, p = driver.cuGraphKernelNodeGetParams(node)
        assert int(err) == 0
        err, name = driver.cuFuncGetName(p.func) if int(p.func) else driver.cuKernelGetName(p.kern)
        assert int(err) == 0
        names.append(name.decode())
    return names


def _values(dtype, E, n, seed):
    rng = np.random.default_rng(seed)
    x = (rng.standard_normal(n) * 2.0 ** rng.integers(-20, 20, n)).astype(dtype)
    x[5 * E] = np.nan
    x[40 * E + 1] = -np.inf
    x[70 * E:71 * E] *= dtype(1e-37 if dtype == np.float32 else 1e-300)
    x[100 * E:140 * E] = 0
    x[110 * E + 3] = -0.0
    x[150 * E:151 * E] = np.finfo(dtype).smallest_subnormal * 5  # no high word in fp64
    x[-E // 2:] = 0  # the partial last block
    return x


@pytest.mark.parametrize("dtype,E,both,only", [(d, *c) for d, cs in CASES.items() for c in cs])
def test_equals_oracle(cuda, dtype, E, both, only):
    f32 = dtype == np.float32
    tdt = torch.float32 if f32 else torch.float64
    n = E * (33000 if f32 else 66000) + E // 2 + 3
    x = _values(dtype, E, n, E)
    t = torch.from_numpy(x).cuda()
    y = torch.empty(n + 32, dtype=tdt, device="cuda")
    for bits in both + only:
        ref = oracle.compress(x, bits, E, canary=0x5C, threads=8)
        buf = torch.full((ref.size + 64,), 0x5C, dtype=torch.uint8, device="cuda")
        names = _kernels(lambda: frsz_b200.compress(t, bits, E, out=buf[:ref.size]))
        assert len(names) == 1 and re.search("k_compress_laneblock", names[0]), (bits, names)
        got = buf.cpu().numpy()
        assert np.array_equal(got[:ref.size], ref) and np.all(got[ref.size:] == 0x5C), bits
        if bits in only:
            continue
        y.fill_(5.0)
        names = _kernels(lambda: frsz_b200.decompress(buf[:ref.size], n, tdt, bits, E, out=y[:n]))
        assert len(names) == 1 and re.search("k_decompress_laneblock", names[0]), (bits, names)
        out = y.cpu().numpy()
        assert np.array_equal(out[:n].view(np.uint8), oracle.decompress(ref, n, dtype, bits, E, threads=8).view(np.uint8)), bits
        assert np.all(out[n:] == 5.0)
