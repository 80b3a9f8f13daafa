"""GPU: products that are redone at a narrower width, in an engine whose error
limit is lowered at set-up: results in pageable memory, whose copy starts before
the outcome is known, and a batch in which only some items are redone."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_CHILD = r"""
import sys
sys.path.insert(0, {root!r}); sys.path.insert(0, {root!r} + "/tests")
import numpy as np
import bluecrunch_b200 as bc
import oracle
from conftest import exact, limbs
bc.init(0, max_round_err=0.02)
redone = 0
for n in (250, 3000, 40000, 300000):
    a, b = limbs(n, n), limbs(n + 1, n - n // 5)
    for square in (False, True):
        y = a if square else b
        c, st = bc.mul(a, None if square else b, square=square, want_stats=True)
        assert st["max_round_err"] < 0.02
        want = exact(a, y, c.size) if n < 4000 else oracle.restated().ntt_mul(a, y, c.size)
        assert np.array_equal(c, want), (n, square)
        redone += st["retries"]
assert redone
items = [(limbs(50 + i, 200 + 971 * i), limbs(90 + i, 300 + 800 * i), None) for i in range(24)]
outs, st = bc.mul_batch(items, want_stats=True)
for (a, b, _), c in zip(items, outs):
    assert np.array_equal(c, exact(a, b, a.size + b.size)), a.size
assert 0 < st["retries"]
print("OK")
"""


def test_redone_products_are_exact():
    p = subprocess.run([sys.executable, "-c", _CHILD.format(root=ROOT)], capture_output=True, text=True, timeout=600)
    assert p.returncode == 0 and p.stdout.strip().endswith("OK"), p.stderr[-2000:]
