"""CPU: the kernels' index arithmetic, compiled for the host from the same
headers and checked against Python integers for every transform length and
digit width, the longest included."""
import os
import random
import shutil
import subprocess

import pytest

import bluecrunch_b200 as bc

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    if not os.path.exists(NVCC):
        pytest.skip("nvcc not available")
    exe = str(tmp_path_factory.mktemp("index") / "index_check")
    subprocess.check_call([NVCC, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a",
                           "-I" + os.path.join(ROOT, "bluecrunch_b200", "csrc"), "-o", exe,
                           os.path.join(ROOT, "tests", "index_host_check.cu")])
    return exe


def run(exe, lines):
    out = subprocess.run([exe], input="\n".join(lines) + "\n", capture_output=True, text=True, check=True).stdout
    return out.strip().split("\n")


def test_words_below_the_imaginary_digits(checker):
    cases = [(M, b) for M in bc.lengths() if M > 5120 for b in range(8, 25)]
    assert max(M for M, _ in cases) == 1 << 30
    for (M, b), line in zip(cases, run(checker, ["P %d %d" % c for c in cases])):
        assert int(line) == M * b // 32, (M, b)


def test_run_records(checker):
    # the carry pass looks for a carry out of the product at the last of them
    cases = [M for M in bc.lengths() if M > 5120]
    for M, line in zip(cases, run(checker, ["N %d" % M for M in cases])):
        assert int(line) == 2 * M // 8, M


def test_words_of_a_run(checker):
    # every word that starts inside a run of 8 digits, the one that straddles
    # into the next run with that run's low bits, at every digit width and at
    # every place a run can have below a word boundary
    rng = random.Random(11)
    cases, want = [], []
    for b in range(8, 25):
        nbits = 8 * b
        for r in list(range(40)) + [rng.randrange(1 << 28) for _ in range(40)]:
            h = rng.choice([0, (1 << nbits) - 1, rng.randrange(1 << nbits)])
            nxt = rng.choice([0, 0xFFFFFFFF, rng.randrange(1 << 32)])
            bit0 = r * nbits
            cases.append("Q %d %d %x %x %x %x" % (bit0, nbits, *((h >> s) & (2 ** 64 - 1) for s in (0, 64, 128)), nxt))
            both = h | nxt << nbits
            want.append([(w, both >> (32 * w - bit0) & 0xFFFFFFFF)
                         for w in range((bit0 + 31) // 32, (bit0 + nbits + 31) // 32)])
    for case, line, e in zip(cases, run(checker, cases), want):
        f = line.split()
        assert [(int(w), int(x, 16)) for w, x in zip(f[::2], f[1::2])] == e, case
