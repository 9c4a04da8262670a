"""The square root of pair_exact.cuh by itself (its reciprocal is checked in
tests/test_pair_exact.py) against __fsqrt_rn on every finite float of 2^-76 or
more, and the significands that its error bound leaves open, counted from the
number theory of its comment.  Where it differs below that range shows why the
range ends there."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def compile_check(out_dir):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    so = os.path.join(out_dir, "libroot_check.so")
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_103a,code=sm_103a", "--fmad=false",
                    "-prec-div=true", "-prec-sqrt=true", "-Xcompiler", "-fPIC", "-shared", "-I",
                    os.path.join(REPO, "include"), os.path.join(REPO, "tests", "cuda", "root_check.cu"), "-o", so],
                   check=True)
    return so


def test_few_midpoints_lie_within_the_error_bound():
    """k + 1/2 in [2^23, 2^24) within 2^-43 (relative) of the root of a float,
    that is of a multiple of 2^23 below 2^47 and of 2^24 above: two k in every
    2^23 for each even c = k^2 + k modulo that spacing, |c| <= 64."""
    k = np.arange(1 << 23, 1 << 24, dtype=np.uint64)
    kk = k * k + k
    spacing = np.where(kk < (1 << 47), 1 << 23, 1 << 24).astype(np.uint64)
    c = kk % spacing
    near = (c <= 64) | (spacing - c <= 64)
    assert 0 < near.sum() <= 2 * 65
    assert ((kk[near] % 2) == 0).all()


@pytest.mark.gpu
def test_root_equals_the_intrinsic_on_every_input(gpu, tmp_path):
    lib = ctypes.CDLL(compile_check(str(tmp_path)))
    counts = (ctypes.c_ulonglong * 4)()
    lib.risltc_test_root.argtypes = [ctypes.c_void_p, ctypes.c_float]
    assert lib.risltc_test_root(counts, -0.0) == 0
    bad, checked, below, largest = counts
    print("in range %d of %d differ; below it %d, the largest %s" %
          (bad, checked, below, np.array([largest], np.uint32).view(np.float32)[0]))
    assert checked == 2 * (0x7f7fffff - 0x19800000 + 1) and bad == 0
    assert largest < 0x19800000
