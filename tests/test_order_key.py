"""The laws' comparisons on the integer pipe against the plain ones, on the CPU:
zeros, denormals, infinities and NaN of either sign."""
import ctypes
import os
import shutil
import struct
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_every_pair(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    out = str(tmp_path / "liborderkey.so")
    cmd = ["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-D__device__=", "-D__host__=", "-D__forceinline__=inline",
           "-I" + os.path.join(ROOT, "liggghts-inl_gb300", "csrc"), "-I/usr/local/cuda/include",
           os.path.join(ROOT, "tests", "order_key_check.cpp"), "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    L = ctypes.CDLL(out)
    mag = [0, 1, 0xfffffffffffff, 0x10000000000000, 0x3fefffffffffffff, 0x3ff0000000000000, 0x3ff0000000000001,
           0x7fefffffffffffff, 0x7ff0000000000000, 0x7ff8000000000000, 0x7fffffffffffffff]
    rng = np.random.default_rng(3)
    mag += [int(v) for v in rng.integers(0, 0x7fefffffffffffff, 200)]
    x = np.array([struct.unpack("<d", struct.pack("<Q", m | s))[0] for m in mag for s in (0, 1 << 63)])
    assert L.check_order(x.ctypes.data_as(ctypes.c_void_p), len(x)) == 0
