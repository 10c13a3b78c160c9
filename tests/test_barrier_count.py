"""The grid barrier of the fused step kernel, on the CPU: its arithmetic
(barrier_count.cuh, the kernel's own) through every order in which blocks can
arrive and poll, a block that polls late among them.  Every block has to take
each step's movement flags, and the count has to be the same in all of them."""
import ctypes
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    out = str(tmp_path_factory.mktemp("barrier") / "libbarriercheck.so")
    cmd = ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-D__device__=", "-D__host__=",
           "-I" + os.path.join(ROOT, "liggghts-inl_gb300", "csrc"),
           os.path.join(ROOT, "tests", "barrier_count_check.cpp"), "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    L = ctypes.CDLL(out)
    L.check_barrier.restype = ctypes.c_long
    L.check_barrier.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_ulonglong, ctypes.POINTER(ctypes.c_long)]
    return L


# the count as a launch starts it, and where the arrivals and the flags carry
@pytest.mark.parametrize("start", [0, (1 << 32) - 3, (1 << 48) - 2, (1 << 64) - 3])
@pytest.mark.parametrize("blocks,steps", [(1, 3), (2, 2), (2, 3), (3, 2)])
def test_every_interleaving(lib, blocks, steps, start):
    states = ctypes.c_long()
    assert lib.check_barrier(blocks, steps, start, ctypes.byref(states)) == 0
    assert states.value > (1 << (2 * blocks * steps))
