"""CPU: the kernels' index arithmetic, compiled for the host from the same
headers and checked against Python integers for every transform length and
digit width, the longest included."""
import os
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
