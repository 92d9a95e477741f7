"""The launch path's own size arithmetic equals the library's, and what is out
of range is refused with the library's message."""
import numpy as np
import pytest

import frsz_b200
from frsz_b200 import codec


@pytest.mark.parametrize("dtype,code", [(np.float32, 0), (np.float64, 1)])
def test_size_equals_library(dtype, code):
    for bits in range(4, (64 if code else 32) + 1):
        for E in (1, 2, 3, 5, 7, 8, 12, 31, 32, 100, 256, 1000, 1024, 65535, 65536):
            for n in (0, 1, E - 1, E, E + 1, 255 * E + 3, 256 * E, 10 ** 6 + 7, 2 ** 40 + 1):
                assert codec._size(code, bits, E, n) == frsz_b200.compressed_size(dtype, bits, E, n), (bits, E, n)


@pytest.mark.parametrize("code,bits,E,match", [(0, 33, 32, "number of bits: 33"), (1, 65, 32, "number of bits: 65"),
                                               (1, 3, 32, "number of bits: 3"), (1, 32, 0, "block size: 0"),
                                               (0, 16, 65537, "block size: 65537")])
def test_refusals(code, bits, E, match):
    with pytest.raises(frsz_b200.Frsz2Error, match=match):
        codec._size(code, bits, E, 1000)


def test_negative_length_is_the_librarys():
    # ctypes passes -1 as 2^64 - 1, whose size no buffer has
    assert codec._size(1, 32, 32, -1) == frsz_b200.compressed_size(np.float64, 32, 32, -1)
