"""GPU: row kernels at splits named here, whatever the tuned table prefers, so
that each kernel is the one that runs: 256-point rows inside three levels
(k5_rows), rows of 1024 points a warp each (k2_rows_w1024) and, with
BC_ROWS_WARP=0, on the block kernel (k2_rows<1024>).  Products with operands
longer than half of the transform, and squares."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))

_CHILD = r"""
import sys
sys.path.insert(0, {root!r}); sys.path.insert(0, {tests!r})
import numpy as np
import bluecrunch_b200 as bc
import oracle
from conftest import limbs
bc.init(0)
R = oracle.restated()
M, L1, L2, Lr = {split!r}
assert (3, L1, L2, Lr) in bc.shape_candidates(M)
bc.set_shape(M, L1, L2, Lr)
bc.force_plan(M, 16)
n = M - 3
for al in (n // 2, n - n // 9):
    a, b = limbs(M + al, al), limbs(M + 1, n - al)
    c, st = bc.mul(a, b, want_stats=True)
    assert st["fft_points"] == M
    assert np.array_equal(c, R.ntt_mul(a, b, n)), al
a = limbs(M + 2, n // 2)
assert np.array_equal(bc.mul(a, square=True), R.ntt_mul(a, a, 2 * a.size))
print("OK")
"""


@pytest.mark.parametrize("warp", ["1", "0"])
@pytest.mark.parametrize("split", [(1 << 21, 128, 64, 256), (1 << 22, 64, 64, 1024)])
def test_split(split, warp):
    p = subprocess.run([sys.executable, "-c", _CHILD.format(root=os.path.dirname(HERE), tests=HERE, split=split)],
                       env=dict(os.environ, BC_ROWS_WARP=warp), capture_output=True, text=True, timeout=600)
    assert p.returncode == 0 and p.stdout.strip().endswith("OK"), p.stderr[-2000:]
