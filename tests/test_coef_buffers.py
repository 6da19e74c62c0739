"""Coefficients are read in place where an image's components lie back to back in memory, and put together otherwise: what a
call reads is always CoefImage.flat()."""

import ctypes

import numpy as np
import pytest

import rcg


def _image(arrs):
    comps = [rcg.CoefComponent(i + 1, 1, 1, 0, 1, a.size // 64, a) for i, a in enumerate(arrs)]
    return rcg.CoefImage(8, 8, comps, np.ones((2, 64), np.uint8))


def _cuts(a):
    return [a[:128], a[128:192], a[192:]]


_BASE = np.arange(256, dtype=np.int16) - 100


@pytest.mark.parametrize("arrs,in_place", [
    (_cuts(_BASE.copy()), True),
    ([_BASE.copy()], True),
    ([c.copy() for c in _cuts(_BASE)], None),                    # wherever the allocator put them
    (_cuts(_BASE.copy())[::-1], False),                          # in another order
    ([_BASE.copy()[:64], _BASE.copy()[128:192]], None),
    (_cuts(np.repeat(_BASE, 2)[::2]), False),                    # strided
    (_cuts(_BASE.astype(np.int32)), False),
    (_cuts(_BASE.astype(">i2")), False),
])
def test_what_a_call_reads_is_flat(arrs, in_place):
    ci = _image(arrs)
    keep, at, count = ci._joined()
    want = ci.flat()
    assert count == want.size
    got = np.ctypeslib.as_array(ctypes.cast(at, ctypes.POINTER(ctypes.c_int16)), (count,))
    assert np.array_equal(got, want)
    if in_place is not None:
        assert (at == arrs[0].ctypes.data) == in_place
    del keep


def test_no_components_are_refused_as_before():
    with pytest.raises(ValueError):
        _image([])._joined()
