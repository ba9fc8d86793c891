"""Tile rules of the grouped planner, on the host."""
import ctypes

import numpy as np

import plfft


def _smooth(top):
    out = [1]
    for p in (2, 3, 5, 7, 11, 13):
        for v in list(out):
            while v * p <= top:
                v *= p
                out.append(v)
    return out


def _splits(lengths):
    f = plfft.lib().plfft_b200_group_splits
    m, how = np.asarray(lengths, np.int64), np.zeros(len(lengths), np.uint8)
    f.argtypes, f.restype = [ctypes.c_void_p, ctypes.c_int64, ctypes.c_void_p], None
    f(m.ctypes.data, m.size, how.ctypes.data)
    return how


def test_four_step_lengths_have_a_split():
    """Every length m = a b up to 2^26 with smooth factors up to 8192; larger
    tiles only where no pair fits the usual one."""
    has = set(_smooth(8192))
    products = np.array([m for m in _smooth(1 << 26) if m > 4096 and
                         any(m % a == 0 and m // a in has for a in has if 1 < a < m)])
    how = _splits(products)
    assert products[how == 0].size == 0
    assert list(_splits([3557763, 1 << 25, 1 << 26, 1 << 24, 65536, 6561])) == [2, 2, 2, 1, 1, 1]
