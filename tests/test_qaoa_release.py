"""What the batched passes read after they hand a buffer back to the staging warps.

tests/emu/release.cpp overwrites an item's amplitudes, phase table and record at every thread's release; no
thread's result may change, and every thread releases each item exactly once (the staging warps count the
arrivals).  Every chunk size of the GPU kernels, every number of bits that a high item mixes, and the low,
middle and measuring passes."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "emu", "release.cpp")
CUH = os.path.join(HERE, "..", "orkan_b200", "csrc", "cuda")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("emu") / "librelease.so")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I" + os.path.join(cuda, "include"), SRC, "-o", out],
                   check=True)
    return C.CDLL(out)


# threads per item of the kernels: 2^C / 16.  High items mix n - C bits: one set per thread from 4 on.
SHAPES = [(11, n) for n in (12, 14, 15, 16, 19)] + [(12, n) for n in (13, 15, 16, 17)] + [(13, 17)]


@pytest.mark.parametrize("log_chunk,n", SHAPES)
@pytest.mark.parametrize("byte_cost", [1, 0])
def test_nothing_is_read_after_the_release(lib, log_chunk, n, byte_cost):
    p = 3
    for j in range(p + 1):
        late, count = C.c_uint(), C.c_uint()
        rc = lib.emu_qaoa_release(n, log_chunk, byte_cost, p, j, (1 << log_chunk) // 16, C.byref(late), C.byref(count))
        assert rc == 0
        assert late.value == 0, f"pass {j}: threads that read a buffer they had released"
        assert count.value == 0, f"pass {j}: threads that do not release once"
