"""The launch path's size arithmetic takes the integer types that the library call
takes -- numpy's of every width, torch's -- with the library's result, and a
buffer too short for a numpy length is refused."""
import ctypes

import numpy as np
import pytest
import torch

import frsz_b200
from frsz_b200 import codec

INTS = [np.int8, np.uint8, np.int16, np.uint16, np.int32, np.uint32, np.int64, np.uint64,
        lambda v: torch.tensor(v), bool]


@pytest.mark.parametrize("dtype,code", [(np.float32, 0), (np.float64, 1)])
def test_equals_library(dtype, code):
    for k, of in enumerate(INTS[:-1]):
        for bits, E, n in ((16, 32, 100), (21, 5, 1), (32, 127, 120), (9, 100, 0)):
            want = frsz_b200.compressed_size(dtype, bits, E, n)
            for args in ((of(bits), E, n), (bits, of(E), n), (bits, E, of(n)), (of(bits), of(E), of(n))):
                got = codec._size(code, *args)
                assert type(got) is int and got == want, (k, args)
    assert codec._size(code, 16, 32, True) == frsz_b200.compressed_size(dtype, 16, 32, 1)


def test_long_lengths_do_not_wrap():
    for n in (np.int32(1 << 28), np.int32((1 << 31) - 1), np.uint32((1 << 32) - 1), np.int64(1 << 40)):
        for bits, E in ((64, np.int32(32)), (np.uint8(64), np.int16(1024)), (64, 32)):
            assert codec._size(1, bits, E, n) == frsz_b200.compressed_size(np.float64, int(bits), int(E), int(n))


def test_short_buffer_is_refused(monkeypatch):
    monkeypatch.setattr(codec, "_require_cuda", lambda t, what: None)  # the check stands before any launch
    with pytest.raises(frsz_b200.Frsz2Error, match="needs 2214592768"):
        frsz_b200.decompress(torch.zeros(4096, dtype=torch.uint8), np.int32(1 << 28), torch.float64, 64, 32)


@pytest.mark.parametrize("args", [(16.0, 32, 100), (16, 32.0, 100), (16, 32, 100.0), ("16", 32, 100)])
def test_other_types_are_refused(args):
    with pytest.raises(ctypes.ArgumentError):
        codec._size(1, *args)
