"""The quantisers' table: under its reciprocal the plain product of every value of a block converts as the quotient does. No GPU is needed."""
import ctypes

import numpy as np

from bitnet_nvfp4_b200 import lib

CODES, SCALES, BLOCKS = 128 * 128, 128, 128 * 8


def _e2m1(x):
    a = np.abs(x)
    c = np.zeros(a.shape, dtype=np.uint8)
    for limit, inclusive in ((0.25, False), (0.75, True), (1.25, False), (1.75, True), (2.5, False), (3.5, True), (5.0, False)):  # ties to even
        c += (a >= limit) if inclusive else (a > limit)
    return c


def test_products_convert_as_quotients():
    table = np.full(CODES + SCALES + BLOCKS, 0xcc, dtype=np.uint8)
    fill = getattr(lib.load(), "_ZN4bnf414fill_quant_lutEPh")
    fill.argtypes, fill.restype = [ctypes.c_void_p], ctypes.c_bool
    assert fill(table.ctypes.data)
    entries = table[CODES + SCALES:].reshape(128, 8)
    rcp, byte = entries[:, :4].copy().view(np.float32)[:, 0], entries[:, 4:].copy().view(np.uint32)[:, 0]
    assert np.array_equal(byte, table[CODES:CODES + SCALES])
    n = np.arange(128, dtype=np.float32)
    for amax in range(128):
        e, m = int(byte[amax]) >> 3, int(byte[amax]) & 7
        scale = np.float32(m / 512 if e == 0 else (1 + m / 8) * 2.0 ** (e - 7))
        assert abs(scale - (amax / 6 or 1)) <= (amax / 6 or 1) / 16
        want = _e2m1(n / scale)
        assert np.array_equal(table[128 * amax:128 * amax + 128], want)
        assert np.array_equal(_e2m1(n[:amax + 1] * rcp[amax]), want[:amax + 1]), amax
