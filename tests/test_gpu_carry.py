"""GPU: the carry pass (k_carry, csrc/bc_kernels.cuh) where carry maps are not
constant, against exact integers: runs of zeros and of ones inside a tile of
1024 runs, across tile edges and over many tiles, carries that pass through all
of them, results that are cut, zero-extended or start off a 16-byte boundary,
at width 16 (the specialised form) and others."""
import numpy as np
import pytest
import torch

import bluecrunch_b200 as bc
from conftest import exact, limbs

pytestmark = pytest.mark.gpu


def _ones(n):
    return np.full(n, 0xFFFFFFFF, dtype=np.uint32)


def _spikes(n, *at):
    x = np.zeros(n, dtype=np.uint32)
    for k in at:
        x[k] = 1
    x[-1] = 1
    return x


def _pairs(n):
    """Operands whose product holds zeros or ones over many runs."""
    low = limbs(n, n)
    low[: n // 2] = 0  # the product's lower half: zeros
    block = np.concatenate([_ones(n // 2), np.zeros(n // 4, dtype=np.uint32), _ones(n - n // 2 - n // 4)])
    return [(_ones(n), _ones(n)),            # (2^N - 1)^2: zeros below, ones above
            (_ones(n), _spikes(n, 0)),       # (2^N - 1)(2^K + 1): ones, a carry through all of them
            (_spikes(n, 0, n // 3), _spikes(n, 7, n // 2)),
            (low, low), (block, _ones(n)), (block, limbs(n + 1, n))]


@pytest.mark.parametrize("n", [5000, 8192, 70001])
@pytest.mark.parametrize("b", [8, 13, 16])
def test_runs_of_zeros_and_ones(gpu, n, b):
    need = (2 * n * 32 + b - 1) // b / 2
    M = next(m for m in bc.lengths() if m >= max(need + 1, 8192))
    bc.force_plan(M, b)
    try:
        for x, y in _pairs(n):
            for CL in (2 * n, 2 * n - 4097, 2 * n + 11):
                got, st = bc.mul(x, y, CL=CL, want_stats=True)
                assert st["fft_points"] == M and st["width"] == b
                assert np.array_equal(got, exact(x, y, CL)), (n, b, CL)
    finally:
        bc.force_plan(0, 0)


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_result_off_a_16_byte_boundary(gpu, shift):
    n = 20000
    x, y = limbs(71, n), limbs(72, n)
    a, b = (torch.from_numpy(v.view(np.int32)).cuda() for v in (x, y))
    for width in (0, 16):
        buf = torch.zeros(2 * n + 8, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        bc.force_width(width)
        try:
            bc.mul(a, b, CL=2 * n, out=buf[shift:])
        finally:
            bc.force_width(0)
        got = buf.cpu().numpy().view(np.uint32)
        assert np.array_equal(got[shift:shift + 2 * n], exact(x, y, 2 * n)), (shift, width)
        assert not got[:shift].any() and not got[shift + 2 * n:].any()
