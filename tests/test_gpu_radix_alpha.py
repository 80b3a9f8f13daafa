"""GPU: conversion leaves (bc_gpu_radix_leaves) whose window drops more than one
limb a round (alpha of 1 and more) or none, against the rounds restated: the
window [floor(alpha (i-1)), n] is multiplied by 10^9, its top limb zero before,
and limb n is the digit; a window that has passed limb n gives zeros, in a time
that does not grow with alpha."""
import ctypes
import math
import time

import numpy as np
import pytest

import oracle
import bluecrunch_b200 as bc
from test_gpu_radix_leaves import Leaf

pytestmark = pytest.mark.gpu


def _rounds(y, n, k, alpha):
    t, s = [int(v) for v in y] + [0], [0] * k
    for i in range(1, k + 1):
        lo = 0 if i == 1 else min(n + 1, max(0, math.floor(alpha * (i - 1))))
        if i > 1:
            t[n] = 0
        elif len(y) > n:
            t[len(y)] = 0
        c = 0
        for j in range(lo, n + 1):
            v = t[j] * 1000000000 + c
            t[j] = v & 0xFFFFFFFF
            c = v >> 32
        s[k - i] = t[n]
    return np.array(s, dtype=np.uint32)


@pytest.mark.parametrize("alpha", [-2.0, 0.0, 0.5, 1.0, 1.7, 31.5, 33.0, 500.0, 1e9, 1e300])
@pytest.mark.parametrize("n,k", [(1, 3), (33, 40), (700, 70)])
def test_any_alpha(gpu, n, k, alpha):
    ys = [oracle.random_limbs(77 + n, n), np.full(n, 0xFFFFFFFF, dtype=np.uint32)]
    arr, outs = (Leaf * 2)(), [np.zeros(k, dtype=np.uint32) for _ in ys]
    for i, y in enumerate(ys):
        arr[i] = Leaf(y.ctypes.data, n, n, k, outs[i].ctypes.data)
    fn = bc._lib().bc_gpu_radix_leaves
    t0 = time.perf_counter()
    assert fn(ctypes.cast(arr, ctypes.c_void_p), 2, ctypes.c_double(alpha)) == 0
    assert time.perf_counter() - t0 < 1.0
    for y, got in zip(ys, outs):
        assert np.array_equal(got, _rounds(y, n, k, alpha))
