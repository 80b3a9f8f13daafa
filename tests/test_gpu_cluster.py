"""GPU: products of the shortest transforms (one cluster of CTAs each,
csrc/bc_cluster.cuh) against exact integers, at every transform length: full
and nearly full lengths, operands longer than half of the transform (digits in
the imaginary part), squares, carries through every run, results cut and
zero-extended, and batches of more products than clusters fit."""
import numpy as np
import pytest

import bluecrunch_b200 as bc
from conftest import exact, limbs

pytestmark = pytest.mark.gpu

LENGTHS = [256, 512, 768, 1024, 1280, 1536, 2048, 2560, 3072, 4096, 5120]


def _most(M, b):
    """The most limbs of two operands whose digits of b bits fill M points."""
    return (2 * M * b) // 32 - 1


@pytest.mark.parametrize("M", LENGTHS)
@pytest.mark.parametrize("b", [8, 13, 19])
def test_every_length(gpu, M, b):
    n = _most(M, b)
    cases = [(n // 2, n - n // 2), (1, n - 1), (n - n // 5, n // 5), (n // 3, n // 2 | 1), (7, 1)]
    bc.force_plan(M, b)
    try:
        for k, (al, bl) in enumerate(cases):
            x, y = limbs(1000 * M + k, al), limbs(2000 * M + k, bl)
            for CL in (al + bl, max(1, (al + bl) // 2 | 1), al + bl + 37):
                got, st = bc.mul(x, y, CL=CL, want_stats=True)
                assert st["fft_points"] == M and st["width"] == b
                assert np.array_equal(got, exact(x, y, CL)), (M, b, al, bl, CL)
        x = limbs(3000 * M, n // 2)
        assert np.array_equal(bc.mul(x, square=True), exact(x, x, 2 * x.size))
        # all ones: every run passes a carry on; a lone top bit: zero runs
        ones = np.full(n // 2, 0xFFFFFFFF, dtype=np.uint32)
        assert np.array_equal(bc.mul(ones, square=True), exact(ones, ones, 2 * ones.size))
        top = np.zeros(n // 2, dtype=np.uint32)
        top[-1] = 0x80000000
        assert np.array_equal(bc.mul(top, ones), exact(top, ones, 2 * ones.size))
    finally:
        bc.force_plan(0, 0)


def test_batch_beyond_the_resident_clusters(gpu):
    rng = np.random.default_rng(5)
    items = []
    for k in range(400):
        al, bl = (int(v) for v in rng.integers(1, 700, 2))
        items.append((limbs(10 * k, al), limbs(10 * k + 1, bl) if k % 3 else None, None))
    for (x, y, _), got in zip(items, bc.mul_batch(items)):
        y = x if y is None else y
        assert np.array_equal(got, exact(x, y, x.size + y.size)), (x.size, y.size)
