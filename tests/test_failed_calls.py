"""CPU: a product call that fails half way returns with nothing in flight.

The library's host code runs against a stand-in for the CUDA runtime
(tests/fake_cudart.c, preloaded in child processes) that keeps copies and
kernels in flight until something waits for them and can make the n-th launch,
copy or pinned allocation fail.  Whatever a failing call has enqueued reads the
caller's arrays and writes memory that the next call uses, so nothing may be
pending when it returns."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    if not os.path.exists(os.path.join(CUDA_INC, "cuda_runtime_api.h")):
        pytest.skip("CUDA headers not available")
    so = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    subprocess.check_call(["gcc", "-std=gnu11", "-O1", "-w", "-shared", "-fPIC", "-I" + CUDA_INC, "-o", so,
                           os.path.join(ROOT, "tests", "fake_cudart.c")])
    return so


_CHILD = r"""
import ctypes, sys
sys.path.insert(0, {root!r})
import bluecrunch_b200 as bc
fake = ctypes.CDLL({so!r})
LAUNCH, COPY, HOSTALLOC = 0, 1, 2
bc.init(0)
lib = bc._lib()
keep = []
def memory(kind, limbs):
    p = ctypes.c_void_p()
    if kind == "pageable":
        keep.append((ctypes.c_uint32 * limbs)())
        return ctypes.addressof(keep[-1])
    assert (fake.cudaHostAlloc(ctypes.byref(p), ctypes.c_size_t(4 * limbs), 0) if kind == "pinned" else
            fake.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(4 * limbs))) == 0
    return p.value
def batch(kind, lens):
    d = (bc.MulDesc * len(lens))()
    for i, (al, bl) in enumerate(lens):
        d[i] = bc.MulDesc(memory(kind, al + bl), al + bl, memory(kind, al), al, memory(kind, bl), bl)
    return d
def call(d, kind=-1, nth=0):
    fake.fake_fail(kind, nth)
    r = lib.bc_gpu_mul_batch(d, len(d), None)
    assert r in (-3, -4), r  # a CUDA call failed; got through (no kernel ran)
    return r
{body}
print("DONE")
"""


def _child(fake, body):
    p = subprocess.run([sys.executable, "-c", _CHILD.format(root=ROOT, so=fake, body=body)],
                       env=dict(os.environ, LD_PRELOAD=fake), capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and p.stdout.strip().endswith("DONE"), p.stdout[-1500:] + p.stderr[-3000:]


# one large product from pinned memory (B crosses on a stream of its own), a
# short one, pageable and device operands, several classes on several streams
LENS = [("pinned", [(1 << 21, 1 << 20)]), ("pinned", [(700, 600)]), ("pageable", [(40000, 30000)]),
        ("device", [(40000, 30000)]), ("pinned", [(300, 200), (5000, 4000), (70000, 60000), (70000, 60001)])]


@pytest.mark.parametrize("kind,lens", LENS)
def test_nothing_in_flight_after_a_failing_call(fake, kind, lens):
    _child(fake, """
d = batch(%r, %r)
# no kernel runs here, so no outcome is ever written: the call that gets through returns a timeout
assert call(d, HOSTALLOC, 0) == -3 and fake.fake_pending() == 0, "first pinned allocation"
for what in (COPY, LAUNCH):
    nth = 0
    while call(d, what, nth) != -4:
        assert fake.fake_pending() == 0, (what, nth, fake.fake_pending())
        nth += 1
    assert fake.fake_pending() == 0 and fake.fake_calls(what) <= nth and (nth or what == COPY)
""" % (kind, lens))


def test_zeros_of_an_empty_operand_are_there_when_the_call_returns(fake):
    _child(fake, """
for other in ([], [(300, 200)]):
    d = batch("device", [(0, 500)] + other)
    fake.fake_fail(-1, 0)
    assert lib.bc_gpu_mul_batch(d, len(d), None) == (-4 if other else 0)
    assert fake.fake_pending() == 0, other
""")


def test_kernel_times_after_a_failed_call(fake):
    # the failed call's events are not read with the next call's (there are
    # no entries for them)
    _child(fake, """
d = batch("device", [(40000, 30000)])
bc.time_kernels(True)
assert call(d) == -4
n = fake.fake_calls(LAUNCH)
fake.fake_spans()
assert call(d) == -4 and fake.fake_spans() == n + 1
assert call(d, LAUNCH, n - 1) == -3 and fake.fake_spans() == 0
assert call(d) == -4 and fake.fake_spans() == n + 1
assert len(bc.kernel_times()) == n
""")


@pytest.mark.parametrize("what", ["small", "leaves", "series", "text", "noalloc"])
def test_nothing_in_flight_after_other_failing_calls(fake, what):
    # every copy and launch of these calls fails in turn; without kernels their
    # results mean nothing, so any end that is not a CUDA error will do
    _child(fake, """
what = %r
lib.bc_gpu_mul_noalloc.argtypes = None
if what == "small":
    d = batch("pageable", [(100, 90)] * 40)
    f = lambda: lib.bc_gpu_mul_small_batch(d, len(d))
elif what == "leaves":
    import numpy as np
    class Leaf(ctypes.Structure):
        _fields_ = [("y", ctypes.c_void_p), ("len", ctypes.c_size_t), ("n", ctypes.c_size_t), ("k", ctypes.c_size_t),
                    ("s", ctypes.c_void_p)]
    l = (Leaf * 3)(*[Leaf(memory("pageable", 50), 50, 50, 40, memory("pageable", 40)) for _ in range(3)])
    f = lambda: lib.bc_gpu_radix_leaves(ctypes.cast(l, ctypes.c_void_p), 3, ctypes.c_double(0.93))
elif what == "series":
    p, q = ctypes.POINTER(ctypes.c_uint32)(), ctypes.POINTER(ctypes.c_uint32)()
    pl, ql = ctypes.c_size_t(), ctypes.c_size_t()
    f = lambda: lib.bc_gpu_e_series(0, 5000, ctypes.byref(p), ctypes.byref(pl), ctypes.byref(q), ctypes.byref(ql))
elif what == "text":
    import os
    fd = os.open("/dev/null", os.O_WRONLY)
    x = memory("pageable", 5000)
    f = lambda: lib.bc_gpu_decimal_write(ctypes.c_void_p(x), ctypes.c_size_t(4999), ctypes.c_size_t(5000),
                                         ctypes.c_size_t(45000), fd, ctypes.c_longlong(0))
else:
    c, a, b = memory("device", 9000), memory("device", 5000), memory("device", 4000)
    S = ctypes.c_size_t
    f = lambda: lib.bc_gpu_mul_noalloc(ctypes.c_void_p(c), S(9000), ctypes.c_void_p(a), S(5000), ctypes.c_void_p(b),
                                       S(4000), None)
failed = 0
for kind in (COPY, LAUNCH):
    for nth in range(40):
        fake.fake_fail(kind, nth)
        r = f()
        failed += r == -3
        assert r == -3 or fake.fake_calls(kind) <= nth, (kind, nth, r)
        if r == -3:
            assert fake.fake_pending() == 0, (kind, nth, fake.fake_pending())
assert failed >= 2, failed
""" % what)
