"""CPU: which kernel a class of short products runs, on the stand-in for the
CUDA runtime (tests/fake_cudart.c) with room for 16 clusters: a cluster of CTAs
each while the class is one round of them (two from 2,048 points on), else one
CTA each.  The grid of the launch tells: whole clusters, or a CTA per product."""
import pytest

import bluecrunch_b200 as bc
from test_failed_calls import _child, fake  # noqa: F401


@pytest.mark.parametrize("M", [256, 512, 768, 1024, 1280, 1536, 2048, 2560, 3072, 4096, 5120])
def test_rounds(fake, M):  # noqa: F811
    nc, most = (8 if M % 512 == 0 else 4), (32 if M >= 2048 else 16)
    _child(fake, """
w, M = %d, %d
for n in (1, 2, 15, 16, 17, 31, 32, 33, 74, 147):
    assert lib.bc_gpu_force_plan(M, w) == 0
    d = batch("device", [(M * w // 32 - 1, M * w // 32 - k %% 3) for k in range(n)])
    fake.fake_fail(-1, 0)
    # a forced width accepts any error, but no kernel ran: a timeout
    assert lib.bc_gpu_mul_batch(d, n, None) == -4
    assert fake.fake_calls(LAUNCH) == 1
    assert fake.fake_last_grid() == (%d * min(n, 16) if n <= %d else n), (n, fake.fake_last_grid())
""" % (16, M, nc, most))
