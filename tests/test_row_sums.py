"""The rows' sums of the anchor iteration and its adjoint, compiled for the host, against 64 bits."""
import ctypes as C
import math
import os
import shutil
import subprocess

import numpy as np
import pytest
from conftest import PKG

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def native(tmp_path_factory):
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    if not shutil.which("g++") or not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("no host compiler or no CUDA headers")
    so = str(tmp_path_factory.mktemp("native") / "sums_host.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-w", "-ffp-contract=off", "-fPIC", "-shared",
                           "-I" + os.path.join(PKG, "csrc"), "-I" + cuda, os.path.join(HERE, "native", "sums_host.cpp"),
                           "-o", so])
    return C.CDLL(so)


def _lanes32(x):
    """The sum of x with 32 lanes, a plain FP32 sum each, and a butterfly."""
    m = -(-len(x) // 32) * 32
    s = np.zeros(32, np.float32)
    for r in np.concatenate([x, np.zeros(m - len(x), np.float32)]).reshape(-1, 32):
        s = s + r
    while len(s) > 1:
        s = s[: len(s) // 2] + s[len(s) // 2 :]
    return float(s[0])


@pytest.mark.parametrize("lanes,per", [(8, 8), (16, 4)])  # 16-bit and 32-bit links
@pytest.mark.parametrize("n", [60, 640, 1300])
def test_adjoint_row_sums_are_as_exact_as_with_32_lanes(native, lanes, per, n):
    f = native.adjoint_row_sum
    f.restype, f.argtypes = C.c_float, [C.c_void_p, C.c_longlong, C.c_int, C.c_int]
    rng = np.random.default_rng(151)
    mine, want = [], []
    for _ in range(1500):
        x = np.ascontiguousarray(1.0 + 0.5 * rng.random(n), np.float32)
        exact = math.fsum(x.astype(np.float64))
        mine.append((f(x.ctypes.data, n, lanes, per) - exact) / exact)
        want.append((_lanes32(x) - exact) / exact)
    rms = lambda e: float(np.sqrt(np.mean(np.square(e))))
    assert rms(mine) <= 1.1 * rms(want)


@pytest.mark.parametrize("lanes,per", [(8, 8), (16, 4)])  # 16-bit and 32-bit links
@pytest.mark.parametrize("n", [1, 7, 60, 640, 7305])
def test_unit_row_sums_hold_twice_the_precision(native, lanes, per, n):
    """Within the bound of a sum in twice FP32's precision, gamma_n^2 of the sum of magnitudes (n u squared,
    and u of a lane's correction where its terms nearly cancel stays below it)."""
    row_sum = native.unit_row_sum
    row_sum.restype, row_sum.argtypes = C.c_double, [C.c_void_p, C.c_longlong, C.c_int, C.c_int]
    rng = np.random.default_rng(150)
    for trial in range(40):
        x = rng.normal(size=n)
        if trial % 4 == 1:
            x = x * 10.0 ** rng.uniform(-4, 0, n)
        elif trial % 4 == 2:
            x = 5.0 + 0.3 * x
        elif trial % 4 == 3:
            x = x - x.mean()
        x = np.ascontiguousarray(x, np.float32)
        exact = math.fsum(x.astype(np.float64))
        size = math.fsum(np.abs(x.astype(np.float64)))
        gamma = (n + 8) * 2.0**-24
        assert abs(row_sum(x.ctypes.data, n, lanes, per) - exact) <= max(gamma * gamma, 2.0**-46) * size
