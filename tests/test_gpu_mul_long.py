"""GPU: products of 2^28 limbs with one operand of more digits than the
transform has points (its imaginary parts start 2^27 words into it), where the
digit positions in bits no longer fit 32 bits.  Both forms of the outer forward
pass (L1 = 256 and 512); checked modulo four primes."""
import numpy as np
import pytest

import bluecrunch_b200 as bc
from conftest import limbs

pytestmark = pytest.mark.gpu

M = 1 << 28


@pytest.fixture(scope="module")
def operands():
    # three to one: 3 * 2^27 of the 2^29 digits of 16 bits are A's
    a, b = limbs(2801, 3 << 26), limbs(2802, 1 << 26)
    return a, b, np.zeros(a.size + b.size, dtype=np.uint32)


@pytest.mark.parametrize("L1,L2,Lr", [(256, 256, 4096), (512, 512, 1024)])
def test_imaginary_digits_beyond_2_32_bits(gpu, orc, operands, L1, L2, Lr):
    a, b, c = operands
    bc.set_shape(M, L1, L2, Lr)
    bc.force_plan(M, 16)
    c[:] = 0
    try:
        _, st = bc.mul(a, b, out=c, want_stats=True)
    finally:
        bc.force_plan(0, 0)
        bc.set_shape(M)
        bc._lib().bc_gpu_load_shape_table(bc.SHAPE_FILE.encode())
    assert st["fft_points"] == M and st["width"] == 16 and st["max_round_err"] < 0.25
    assert orc.modcheck(c, a, b, 4)
