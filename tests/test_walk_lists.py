"""Direction lists as users write them -- rounded to a few decimals, of another length than 1 --
walk the reference's staircases: the filtered walk of the tracing kernel, compiled for the host,
against the reference's operations, and on the GPU the line table and staircases against the oracle."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest
from conftest import PKG, REPO

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def native(tmp_path_factory):
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    if not shutil.which("g++") or not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("no host compiler or no CUDA headers")
    so = str(tmp_path_factory.mktemp("native") / "geometry_host.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-w", "-ffp-contract=off", "-fPIC", "-shared",
                           "-I" + os.path.join(PKG, "csrc"), "-I" + os.path.join(REPO, "include"), "-I" + cuda,
                           os.path.join(HERE, "native", "geometry_host.cpp"), "-o", so])
    L = C.CDLL(so)
    L.filtered_walk_differences.argtypes = [C.c_int] * 3 + [C.c_void_p, C.c_longlong, C.c_void_p, C.c_void_p]
    L.wrong_misses.argtypes = [C.c_int] * 3 + [C.c_void_p, C.c_longlong, C.c_void_p]
    L.filtered_walk_differences.restype = L.wrong_misses.restype = C.c_longlong
    return L


def _units(n, seed):
    k = np.random.default_rng(seed).normal(size=(n, 3))
    return k / np.linalg.norm(k, axis=1, keepdims=True)


def _list(kind, n=8, seed=110):
    """n directions, of unit length in FP32, rounded to so many decimals, or of another length."""
    k = _units(n, seed)
    if kind.startswith("decimals"):
        k = np.round(k, int(kind[8:]))
    elif kind.startswith("length"):
        k = k * float(kind[6:])
    return k.astype(np.float32)


LISTS = ["unit", "decimals2", "decimals3", "decimals4", "decimals5", "length0.99", "length0.999", "length1.01",
         "length0.99997", "length1.00003"]


@pytest.mark.parametrize("dims", [(24, 24, 24), (41, 37, 40), (5, 3, 150)])
@pytest.mark.parametrize("kind", LISTS)
def test_filtered_walk_takes_the_reference_steps(orc, native, kind, dims):
    for k in _list(kind):
        if not np.all(np.abs(k) < 1.0):
            continue  # (the rotation of such a direction has no angle)
        valid, inout, _, xyz = orc.trace_direction(dims, 1.0, k)
        at = np.nonzero(valid)[0]
        io, o = np.ascontiguousarray(inout[at], np.int32), np.ascontiguousarray(xyz[at], np.float32)
        assert native.filtered_walk_differences(*dims, k.ctypes.data, len(at), io.ctypes.data, o.ctypes.data) == 0


@pytest.mark.parametrize("k1", [0.8660254, -30.0, 3e3, -2e5, 1e8])
def test_certain_misses_miss(native, k1):
    """Lines through points within a few roundings of the grid's silhouette.  The rotation takes its
    angles from k2 and k3, so a first component of any size is accepted, and the roundings grow with it."""
    dims = (40, 37, 41)
    c = (np.array(dims) - 1) / 2
    rng = np.random.default_rng(111)
    n = 200000
    for k2, k3 in ((0.3, 0.4), (0.5, -0.2), (-0.01, 0.7)):
        k = np.array([k1, k2, k3], np.float32)
        # a point on an edge of the grid, moved along the direction and off it by a few ulp
        at = rng.uniform(-1, 1, (n, 3)) * c
        for a, side in zip(rng.permuted(np.tile(np.arange(3), (n, 1)), axis=1)[:, :2].T, rng.choice([-1, 1], (2, n))):
            at[np.arange(n), a] = side * c[a]
        at += rng.uniform(-60, 60, (n, 1)) * (k / np.linalg.norm(k))
        at *= 1 + rng.integers(-8, 9, (n, 3)) * 2.0**-24
        o = np.ascontiguousarray(at, np.float32)
        assert native.wrong_misses(*dims, k.ctypes.data, n, o.ctypes.data) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["decimals2", "decimals3", "length0.99", "length0.999", "length1.01"])
def test_list_walks_bit_exact(omni, orc, match_lines, kind):
    from test_gpu_parity import _lines_oracle

    dims = (40, 37, 41)
    dirs = _list(kind, n=6)
    with omni.Omni3D(dims, 1e-3, dirs, max_iter=1) as s:
        got = s.line_table().astype(np.int64)
        exp, geo = _lines_oracle(orc, dims, 1.0, dirs)
        at = match_lines(got, exp)
        p = np.zeros(int(np.prod(dims)), np.float32)
        _, count = s.sweep(p, p, p, p)
        for k in range(0, len(exp), 29):
            io, xyz = geo[k]
            ax = orc.walk(dims, io, xyz, dirs[exp[k, 2]])
            assert any(np.array_equal(s.line_steps(i), ax) for i in at[k]), k
    _, expected = orc.sweep(dims, (1e-3, 1e-3, 1e-3), dirs, p, p, p, p, mode=0, precision="f64", nthreads=4)
    np.testing.assert_array_equal(count.reshape(-1), expected.astype(np.float32))  # every line's staircase
