"""The launch shape of the anchor iterations."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest
from conftest import PKG

HERE = os.path.dirname(os.path.abspath(__file__))


def test_shared_memory_iterations_run_in_one_round(tmp_path):
    """A CTA of 1024 threads with the vector in shared memory has an SM for itself: more blocks than the
    152 SMs would wait for a second round, and fill their shared memory again."""
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    if not shutil.which("g++") or not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("no host compiler or no CUDA headers")
    so = str(tmp_path / "links_host.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-w", "-fPIC", "-shared", "-I" + os.path.join(PKG, "csrc"),
                           "-I" + cuda, os.path.join(HERE, "native", "links_host.cpp"), "-o", so])
    f = C.CDLL(so).unit_iter_shape
    f.restype, f.argtypes = None, [C.c_longlong, C.c_void_p]
    out = np.zeros(4, np.int32)
    seen = 0
    for n in [6 * m * m - 12 * m + 8 for m in range(4, 160)] + [16383, 16384, 27648, 27649, 55296, 55297, 110592, 110593]:
        f(n, out.ctypes.data)
        smem, blocks, rows, least = (int(x) for x in out)
        assert least <= rows <= 24 and blocks * rows * (32 if smem else 8) >= n
        if smem:
            seen += 1
            assert blocks <= 152, (n, blocks)
    assert seen > 50
