"""The ray queue's 32-bit cursor near 2^32 rays, on the CPU: wherever the rule
lets a queue use the cursor, the warps' last fetches (of 32 each, the worst case,
one after another past the last ray) leave it without a wrap, and every warp
ends; it lets every count up to 2^31 and beyond use it."""
import ctypes
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    so = str(tmp_path_factory.mktemp("cursor") / "libcursor_check.so")
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-Xcompiler", "-fPIC", "-shared",
                    "-I", os.path.join(REPO, "include"), os.path.join(REPO, "tests", "cuda", "cursor_check.cu"),
                    "-o", so], check=True)
    lib = ctypes.CDLL(so)
    lib.risltc_test_cursor_holds.argtypes = [ctypes.c_uint, ctypes.c_uint]
    return lambda rays, threads: bool(lib.risltc_test_cursor_holds(rays, threads))


def fetches_end(rays, threads):
    """The cursor's last steps as the warps take them, from 33 rays before the
    end: True if every warp sees the end without the cursor wrapping."""
    cursor, warps = (rays - 33) % (1 << 32), threads // 32
    while warps:
        base = cursor
        cursor += 32
        if cursor >= 1 << 32:
            return False
        if base + 32 >= rays:
            warps -= 1
    return True


@pytest.mark.parametrize("threads", [152 * 12 * 128, 132 * 12 * 128, 32])
def test_the_cursor_never_wraps_where_it_is_used(rule, threads):
    top = (1 << 32) - 1
    for rays in (threads + 1, 1 << 31, 3 << 30, top - 2 * threads, top - threads - 32, top - threads - 1, top - threads,
                 top - threads + 1, min(top, top - threads + 33), top - threads // 2, top - 31, top):
        if rule(rays, threads):
            assert fetches_end(rays, threads)
        else:
            assert rays > top - threads
    assert not fetches_end(top, threads)  # what the rule is for
