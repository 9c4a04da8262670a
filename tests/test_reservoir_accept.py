"""The candidate kernel's reservoir test without its division (reservoir_accepts)
against rnd < w / w_sum on 2^28 triples from subnormal to infinite weights:
random numbers of exactly 0 with quotients that underflow, sums within a few
units of the border, both numerics modes."""
import ctypes
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def compile_check(out_dir):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    so = os.path.join(out_dir, "libaccept_check.so")
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_103a,code=sm_103a", "--fmad=false",
                    "-prec-div=true", "-prec-sqrt=true", "-Xcompiler", "-fPIC", "-shared", "-I",
                    os.path.join(REPO, "include"), os.path.join(REPO, "tests", "cuda", "accept_check.cu"), "-o", so],
                   check=True)
    return so


@pytest.mark.gpu
def test_accepts_what_the_division_accepts(gpu, tmp_path):
    lib = ctypes.CDLL(compile_check(str(tmp_path)))
    counts = (ctypes.c_ulonglong * 4)()
    lib.risltc_test_accept.argtypes = [ctypes.c_void_p]
    assert lib.risltc_test_accept(counts) == 0
    exact, fast, zero, accepted = counts
    assert exact == 0 and fast == 0
    assert zero > 1 << 20 and 1 << 24 < accepted < (1 << 28) - (1 << 24)
