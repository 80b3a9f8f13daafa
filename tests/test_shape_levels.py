"""Splits of two levels at the lengths whose built-in split has three (2^20 to
2^21 points): accepted one by one and from a file, and exact on the GPU.  Where
the built-in split has two levels, three are refused."""
import numpy as np
import pytest

import bluecrunch_b200 as bc
from conftest import limbs

TWO = [(5 << 18, 512, 1, 2560), (3 << 19, 512, 1, 3072), (1 << 21, 512, 1, 4096)]


def _reload():
    for M, *_ in TWO:
        bc.set_shape(M)
    bc._lib().bc_gpu_load_shape_table(bc.SHAPE_FILE.encode())


@pytest.mark.parametrize("M,L1,L2,Lr", TWO)
def test_two_levels_above_the_built_in_line(tmp_path, M, L1, L2, Lr):
    lib = bc._lib()
    assert (2, L1, L2, Lr) in bc.shape_candidates(M)
    assert any(c[0] == 3 for c in bc.shape_candidates(M))
    f = tmp_path / "shapes.txt"
    f.write_text("%d %d %d %d\n" % (M, L1, L2, Lr))
    try:
        assert lib.bc_gpu_set_shape(M, L1, L2, Lr) == 0
        assert lib.bc_gpu_check_shapes() == 0
        bc.set_shape(M)
        assert lib.bc_gpu_load_shape_table(str(f).encode()) == 0
        assert lib.bc_gpu_force_plan(M, 16) == 0
        assert bc.plan(M // 2 - 2, M // 2 - 2)["levels"] == 2
    finally:
        bc.force_plan(0, 0)
        _reload()


@pytest.mark.parametrize("M,L1,L2,Lr", [(3 << 18, 64, 64, 192), (1 << 20, 64, 64, 256)])
def test_three_levels_below_it_are_refused(M, L1, L2, Lr):
    assert bc._lib().bc_gpu_set_shape(M, L1, L2, Lr) == -1
    assert all(c[0] == 2 for c in bc.shape_candidates(M))


@pytest.mark.gpu
@pytest.mark.parametrize("M,L1,L2,Lr", TWO)
def test_products_of_such_splits(gpu, orc, M, L1, L2, Lr):
    n = M - 4
    a, b = limbs(M + 1, n - n // 3), limbs(M + 2, n // 3)
    bc.set_shape(M, L1, L2, Lr)
    bc.force_plan(M, 16)
    try:
        got, st = bc.mul(a, b, want_stats=True)
        assert st["fft_points"] == M
        assert np.array_equal(got, orc.ntt_mul(a, b, n))
        s = a[:n // 2]
        assert np.array_equal(bc.mul(s, square=True), orc.ntt_mul(s, s, 2 * s.size))
    finally:
        bc.force_plan(0, 0)
        _reload()
