"""GPU: row passes of 128, 192, 256, 320, 384, 640 and 768 points (k5_rows,
csrc/bc_rows2.cuh) inside two- and three-level transforms, against exact
products: full lengths, operands longer than half of the transform, squares, and
a batch whose items share a transform length (several items, B shared)."""
import numpy as np
import pytest

import bluecrunch_b200 as bc
from conftest import limbs

pytestmark = pytest.mark.gpu

# (M, L1, L2, Lr): every row length with two levels, and with three
SHAPES = [(64 * r, 64, 1, r) for r in (128, 192, 256, 320, 384, 640, 768)] + \
         [(512 * r, 512, 1, r) for r in (128, 192, 256, 320, 384, 640, 768)] + \
         [(64 * 64 * 256, 64, 64, 256), (128 * 64 * 320, 128, 64, 320), (64 * 128 * 384, 64, 128, 384),
          (128 * 128 * 192, 128, 128, 192), (256 * 128 * 128, 256, 128, 128), (64 * 64 * 640, 64, 64, 640), (64 * 64 * 768, 64, 64, 768)]


@pytest.mark.parametrize("M,L1,L2,Lr", SHAPES)
def test_products_and_squares(gpu, orc, M, L1, L2, Lr):
    b = 16
    n = 2 * M * b // 32 - 2
    if (L1, L2, Lr) not in [s[1:] for s in bc.shape_candidates(M)]:
        pytest.skip("the length's built-in shape has another number of levels")
    bc.set_shape(M, L1, L2, Lr)
    bc.force_plan(M, b)
    try:
        for al, bl in ((n // 2, n - n // 2), (n - n // 7, n // 7)):
            x, y = limbs(M + al, al), limbs(M + bl + 1, bl)
            got, st = bc.mul(x, y, want_stats=True)
            assert st["fft_points"] == M
            assert np.array_equal(got, orc.ntt_mul(x, y, al + bl)), (al, bl)
        x = limbs(M + 5, n // 2)
        assert np.array_equal(bc.mul(x, square=True), orc.ntt_mul(x, x, 2 * x.size))
    finally:
        bc.force_plan(0, 0)
        bc.set_shape(M)
        bc.load_shape_table() if hasattr(bc, "load_shape_table") else bc._lib().bc_gpu_load_shape_table(
            bc.SHAPE_FILE.encode())


def test_batch_of_one_length(gpu, orc):
    items = [(limbs(9000 + k, 16000 + 7 * k), limbs(9100 + (k // 2), 15000), None) for k in range(9)]
    for (x, y, _), got in zip(items, bc.mul_batch(items)):
        assert np.array_equal(got, orc.ntt_mul(x, y, x.size + y.size))
