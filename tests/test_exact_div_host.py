"""The division on the FP32 and integer pipes (csrc/ccd_div.h) on the host:
the quotient is the IEEE one for every operand pair and for every reciprocal
estimate within the device instruction's error."""
import ctypes

import numpy as np
import pytest

from hostcheck import build as hb

P = ctypes.c_void_p


def _div(a, b, ulps):
    lib = ctypes.CDLL(hb._build("hc_div", "hostcheck_div.cpp"))
    q = np.zeros_like(a)
    lib.hc_div(a.ctypes.data_as(P), b.ctypes.data_as(P), ctypes.c_int64(a.size), ctypes.c_int(ulps),
               q.ctypes.data_as(P))
    return q


def _significands(rng, n, how):
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    if how == "ones":
        m |= np.uint64(((1 << 52) - 1) & ~0xff)
    elif how == "zeros":
        m &= np.uint64(0xff)
    elif how == "low":  # only the trailing 29 bits, or all but them
        m = np.where(rng.random(n) < 0.5, m & np.uint64(0x1fffffff), m & ~np.uint64(0x1fffffff))
    return m


@pytest.mark.parametrize("ulps", [-1, 0, 1])
@pytest.mark.parametrize("how", ["random", "ones", "zeros", "low", "near", "midpoint"])
def test_quotient_is_exact(how, ulps):
    rng = np.random.default_rng([5, len(how), ulps + 1])
    n = 1_000_000
    bits = []
    for _ in range(2):
        e = rng.integers(523, 1524, n, dtype=np.uint64) << np.uint64(52)
        sign = rng.integers(0, 2, n, dtype=np.uint64) << np.uint64(63)
        bits.append(_significands(rng, n, how) | e | sign)
    a, b = (x.view(np.float64) for x in bits)
    if how == "near":  # quotients next to a power of two
        a = (bits[1] + rng.integers(0, 7, n, dtype=np.uint64) - np.uint64(3)).view(np.float64)
    elif how == "midpoint":  # a nearest to b times a number half-way between two doubles
        b = ((bits[1] & np.uint64((1 << 52) - 1)) | np.uint64(1023 << 52)).view(np.float64)
        q = 1.0 + rng.random(n)
        a = q * b + 2.0 ** -53 * b
    got = _div(np.ascontiguousarray(a), np.ascontiguousarray(b), ulps)
    np.testing.assert_array_equal(got.view(np.uint64), (a / b).view(np.uint64))
