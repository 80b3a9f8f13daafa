"""GPU: conversion leaves whose rounds carry through many limbs (k_radix_leaves
keeps limbs unresolved, csrc/bc_radix.cuh) against the reference's rounds
restated in the oracle: all ones (every digit's carry is in doubt), ones in the
upper or the lower part only, ones that end at a lane's edge (32 limbs), a lone
low bit, and all ones with one limb cleared."""
import math

import numpy as np
import pytest

import oracle
from test_gpu_radix_leaves import ALPHA, _gpu_leaves

pytestmark = pytest.mark.gpu


def _fractions(n):
    ones = np.full(n, 0xFFFFFFFF, dtype=np.uint32)
    out = [ones]
    for cut in sorted({1, 31, 32, 33, 64, n // 2, n - 1}):
        if 0 < cut < n:
            lo, hi, hole = ones.copy(), ones.copy(), ones.copy()
            lo[cut:] = 0
            hi[:cut] = 0
            hole[cut] = 0
            out += [lo, hi, hole]
    bit = np.zeros(n, dtype=np.uint32)
    bit[0] = 1
    top = np.zeros(n, dtype=np.uint32)
    top[-1] = 1
    return out + [bit, top]


@pytest.mark.parametrize("k", [3, 34, 70, 400, 1000])
def test_long_carries(gpu, k):
    n = int(math.floor((k * math.log(1e9) + math.log(4.0) + math.log(1000.0)) / math.log(4294967296.0) + 1))
    cases = [(y, n, k) for y in _fractions(n)]
    for (y, _, _), got in zip(cases, _gpu_leaves(cases)):
        assert np.array_equal(got, oracle.convert_trunc(y, n, k, ALPHA))
