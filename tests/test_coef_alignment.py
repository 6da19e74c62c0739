"""Coefficients at an odd address are put together in an aligned array: a call reads them as 16-bit integers."""

import ctypes

import numpy as np

import rcg


def test_unaligned_coefficients_are_copied():
    raw = np.zeros(2 * 192 + 1, np.uint8)
    raw[1:] = np.arange(192, dtype=np.int16).view(np.uint8)
    a = raw[1:].view(np.int16) if raw.ctypes.data % 2 == 0 else raw[:-1].view(np.int16)
    assert a.ctypes.data % 2 == 1 and not a.flags.aligned
    ci = rcg.CoefImage(8, 8, [rcg.CoefComponent(1, 1, 1, 0, 1, 1, a[:64]), rcg.CoefComponent(2, 1, 1, 1, 1, 2, a[64:])],
                       np.ones((2, 64), np.uint8))
    keep, at, count = ci._joined()
    assert at % 2 == 0 and count == 192
    got = np.ctypeslib.as_array(ctypes.cast(at, ctypes.POINTER(ctypes.c_int16)), (count,))
    assert np.array_equal(got, ci.flat())
    del keep
