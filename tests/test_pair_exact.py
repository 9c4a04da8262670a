"""The paired sequences of pair_exact.cuh (two scalar computations in the
lanes of FADD2 / FFMA2) against CUDA's correctly rounded scalar intrinsics:
the reciprocal square root on every finite float of 2^-76 or more and the edge
integral's rational fit on every float of (0, 1 + 2^-15], in both lanes, and
products, sums and differences of products on random bit patterns.  Exact
numerics may use them only because they are bit-identical there."""
import ctypes
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def compile_check(out_dir):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    so = os.path.join(out_dir, "libpair_check.so")
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_103a,code=sm_103a", "--fmad=false",
                    "-prec-div=true", "-prec-sqrt=true", "-Xcompiler", "-fPIC", "-shared", "-I",
                    os.path.join(REPO, "include"), os.path.join(REPO, "tests", "cuda", "pair_check.cu"), "-o", so],
                   check=True)
    return so


@pytest.mark.gpu
def test_paired_sequences_equal_the_intrinsics_on_every_input(gpu, tmp_path):
    lib = ctypes.CDLL(compile_check(str(tmp_path)))
    counts = (ctypes.c_ulonglong * 5)()
    lib.risltc_test_pairs.argtypes = [ctypes.c_void_p, ctypes.c_float]
    assert lib.risltc_test_pairs(counts, -0.0) == 0
    root, roots, fit, fits, operations = counts
    assert roots == 2 * (0x7f7fffff - 0x19800000 + 1) and root == 0
    assert fits == 2 * 0x3f800100 and fit == 0
    assert operations == 0
