"""Contexts that walk the row-major volume, as grids of 2^30 voxels and contexts without memory for the
skewed copies do: every method, precision and form, against the FP64 oracle or the same call over
skewed copies, and contexts that lose their copies between two calls.  The allocation failure
is a fake one (omni3d_test_copies)."""
import ctypes as C

import numpy as np
import pytest
from test_gpu_parity import TOL_P_PLAIN, TOL_P_SELECT, TOL_PN

from omni3d import synthetic
from omni3d._lib import lib

pytestmark = pytest.mark.gpu

METHODS = ["plain", "select", "weighted", "weighted_fixed_bc", "select_fixed_bc", "mini_curl", "weighted_mini_curl"]
DIMS = (20, 18, 16)


def _copies(s, lose=False):
    f = lib().omni3d_test_copies
    f.restype, f.argtypes = C.c_int, [C.c_void_p, C.c_int]
    return f(s.handle, int(lose))


def _field(orc, dims=DIMS, seed=120):
    f = synthetic.blobs(dims=dims, count=3, sigma_range=(2.0, 5.0), noise=0.05, seed=seed, sphere_radius=3.5)
    curl = orc.curl(dims, f["spacing"], f["ax"], f["ay"], f["az"], f["mask"])
    return f, curl, float(np.percentile(curl[curl > 0], 85))


def _tol(method):
    return TOL_P_PLAIN if method in ("plain", "mini_curl") else TOL_P_SELECT


def _same(a, b, method):
    if method in ("plain", "mini_curl"):  # unit weights: the counts are whole numbers
        np.testing.assert_array_equal(a.count, b.count)
    else:
        assert synthetic.relative_l2(a.count, b.count, gauge="none") < 1e-5
    assert synthetic.relative_l2(a.p, b.p, gauge="none") < 2 * _tol(method)


@pytest.mark.parametrize("option", ["", "bf16", "sweep", "sweep_fp64", "deterministic", "tol"])
@pytest.mark.parametrize("method", METHODS)
def test_row_major_solve(omni, orc, method, option):
    f, curl, thr = _field(orc)
    a = [f[k] for k in ("ax", "ay", "az")]
    opts = {"": {}, "bf16": {"grad": "bf16"}, "sweep": {"solver": "sweep"}, "tol": {"tol": 1e-30, "max_iter": 40},
            "sweep_fp64": {"sweep_fp64": True}, "deterministic": {"deterministic": True}}[option]
    opts = dict(dict(max_iter=4, method=method, threshold=thr, gauge="mean"), **opts)
    with omni.Omni3D(DIMS, f["spacing"], omni.icosphere(3), **opts) as s:
        want = s.solve(*a, curl=curl)
        assert _copies(s, lose=True) == 1
        got = s.solve(*a, curl=curl)  # gives up its copies and starts over
        assert _copies(s) == 0
        _same(got, want, method)
        assert got.stats["iterations"] == want.stats["iterations"]
        _same(s.solve(*a, curl=curl), want, method)  # a row-major context's second solve
    with omni.Omni3D(DIMS, f["spacing"], omni.icosphere(3), **opts) as s:  # row-major from the start
        _copies(s, lose=True)
        _same(s.solve(*a, curl=curl), want, method)
        assert _copies(s) == 0


@pytest.mark.parametrize("method,mode", [("plain", 0), ("select", 1), ("weighted", 2)])
@pytest.mark.parametrize("solver", ["anchor", "sweep"])
def test_row_major_solve_matches_fp64_oracle(omni, orc, method, mode, solver):
    f, curl, thr = _field(orc)
    dirs = omni.icosphere(3)
    with omni.Omni3D(DIMS, f["spacing"], dirs, max_iter=4, method=method, threshold=thr, solver=solver) as s:
        _copies(s, lose=True)
        r = s.solve(f["ax"], f["ay"], f["az"], curl=curl)
        assert _copies(s) == 0
    ep, _ = orc.solve(DIMS, f["spacing"], dirs, f["ax"], f["ay"], f["az"], np.zeros(int(np.prod(DIMS)), np.float32), 4,
                      mode=mode, thr=thr, curl=curl, precision="f64", nthreads=4)
    assert synthetic.relative_l2(r.p, ep, gauge="none") < _tol(method)


def test_row_major_operator_with_signed_curls(omni, orc):
    """A curl with its sign bit set leaves no bit for the anchor flags: ids are gathered instead."""
    f, curl, thr = _field(orc)
    signed = curl.copy()
    signed[::37] *= -1.0
    for method in ("select", "weighted"):
        with omni.Omni3D(DIMS, f["spacing"], omni.icosphere(3), max_iter=3, method=method, threshold=thr) as s:
            want = s.solve(f["ax"], f["ay"], f["az"], curl=signed)
            _copies(s, lose=True)
            _same(s.solve(f["ax"], f["ay"], f["az"], curl=signed), want, method)
            assert _copies(s) == 0


@pytest.mark.parametrize("method,mode", [("plain", 0), ("select", 1), ("weighted", 2)])
@pytest.mark.parametrize("dims", [(2, 3, 5), (31, 33, 32), (65, 5, 7), (4, 64, 33), (33, 3, 66), (48, 50, 47)])
def test_row_major_sweep(omni, orc, dims, method, mode):
    rng = np.random.default_rng(121)
    a = [rng.normal(size=int(np.prod(dims))).astype(np.float32) for _ in range(3)]
    p = rng.normal(size=int(np.prod(dims))).astype(np.float32)
    h, dirs = (1e-3,) * 3, omni.icosphere(3)
    curl = orc.curl(dims, h, *a, np.ones(int(np.prod(dims)), np.float32))
    thr = float(np.percentile(curl, 80))
    epn, ecnt = orc.sweep(dims, h, dirs, *a, p, mode=mode, thr=thr, curl=curl, precision="f64", nthreads=4)
    with omni.Omni3D(dims, h, dirs, max_iter=2, method=method, threshold=thr) as s:
        _copies(s, lose=True)
        for _ in range(2):
            pn, cnt = s.sweep(*a, p, curl=curl)
            assert _copies(s) == 0
            assert synthetic.relative_l2(pn.reshape(-1), epn, gauge="none") < TOL_PN
            assert synthetic.relative_l2(cnt.reshape(-1), ecnt, gauge="none") < TOL_PN
            s.solve(*a, curl=curl)


@pytest.mark.parametrize("method,mode", [("plain", 0), ("select", 1), ("weighted", 2), ("mini_curl", 5),
                                         ("weighted_mini_curl", 6)])
def test_row_major_adjoint(omni, orc, method, mode):
    dims = (13, 11, 10)
    f, curl, thr = _field(orc, dims, 122)
    dirs = omni.icosphere(2)
    g = np.random.default_rng(7).normal(size=int(np.prod(dims))).astype(np.float32)
    exp = orc.adjoint_modes(dims, f["spacing"], dirs, 4, g, mode=mode, thr=thr, curl=curl)
    with omni.Omni3D(dims, f["spacing"], dirs, max_iter=4, method=method, threshold=thr) as s:
        _copies(s, lose=True)
        s.solve(f["ax"], f["ay"], f["az"], curl=curl)
        assert _copies(s) == 0
        for a, b in zip(s.adjoint(g), exp):
            assert synthetic.relative_l2(a, b, gauge="none") < 1e-4


@pytest.mark.parametrize("method", ["plain", "select"])
def test_batch_member_that_loses_its_copies(omni, method):
    """Between two batch solves one member's own solve gives up its copies: the captured graph (plain
    method) no longer fits its buffers."""
    sizes = [(17, 15, 19), (21, 16, 14), (18, 22, 15)]
    fs = [synthetic.blobs(dims=d, count=3, sigma_range=(2.0, 4.0), noise=0.05, seed=123 + i) for i, d in enumerate(sizes)]
    dirs = omni.icosphere(3)
    members = [omni.Omni3D(d, f["spacing"], dirs, max_iter=5, method=method, threshold=1e30) for d, f in zip(sizes, fs)]
    args = [(f["ax"], f["ay"], f["az"]) for f in fs]
    try:
        with omni.Batch(members) as b:
            want, counts, _ = b.solve(args)
            want = [np.array(p) for p in want]
            for lost in (1, 0):
                _copies(members[lost], lose=True)
                members[lost].solve(*args[lost])
                assert _copies(members[lost]) == 0
                for _ in range(2):
                    ps, cs, _ = b.solve(args)
                    for i in range(3):
                        assert synthetic.relative_l2(ps[i], want[i], gauge="none") < 2 * _tol(method)
                        if method == "plain":
                            np.testing.assert_array_equal(cs[i], counts[i])
    finally:
        for s in members:
            s.close()


@pytest.mark.parametrize("method", ["plain", "select"])
def test_adjoint_after_one_that_found_no_memory(omni, orc, method):
    """An adjoint that could not allocate its transposed links leaves nothing of them behind."""
    dims = (13, 11, 10)
    f, curl, thr = _field(orc, dims, 124)
    g = np.random.default_rng(8).normal(size=int(np.prod(dims))).astype(np.float32)
    with omni.Omni3D(dims, f["spacing"], omni.icosphere(2), max_iter=4, method=method, threshold=thr) as s:
        _copies(s, lose=True)
        s.solve(f["ax"], f["ay"], f["az"], curl=curl)
        fail = lib().omni3d_test_no_adjoint_links
        fail.restype, fail.argtypes = None, [C.c_void_p]
        fail(s.handle)
        with pytest.raises(omni.Omni3DError) as e:
            s.adjoint(g)
        assert e.value.code == -4
        after = s.adjoint(g)
    with omni.Omni3D(dims, f["spacing"], omni.icosphere(2), max_iter=4, method=method, threshold=thr) as s:
        s.solve(f["ax"], f["ay"], f["az"], curl=curl)
        for a, b in zip(after, s.adjoint(g)):
            assert synthetic.relative_l2(a, b, gauge="none") < 1e-5


@pytest.mark.parametrize("gauge", ["none", "mean"])
@pytest.mark.parametrize("method", METHODS)
def test_adjoint_gives_up_the_copies_for_memory(omni, orc, method, gauge):
    """Links that find no memory beside the skewed copies find it without them: the adjoint starts over
    row-major, and the solves after it are."""
    torch = pytest.importorskip("torch")
    dims = (13, 11, 10)
    f, curl, thr = _field(orc, dims, 125)
    g = np.random.default_rng(9).normal(size=int(np.prod(dims))).astype(np.float32)
    a = [f[k] for k in ("ax", "ay", "az")]
    fail = lib().omni3d_test_no_adjoint_links
    fail.restype, fail.argtypes = None, [C.c_void_p]
    with omni.Omni3D(dims, f["spacing"], omni.icosphere(2), max_iter=4, method=method, threshold=thr, gauge=gauge) as s:
        first = s.solve(*a, curl=curl)
        want = s.adjoint(g)
        for device in (False, True):
            with omni.Omni3D(dims, f["spacing"], omni.icosphere(2), max_iter=4, method=method, threshold=thr,
                             gauge=gauge) as t:
                t.solve(*a, curl=curl)
                fail(t.handle)
                if device:  # the gradient's own memory takes the result
                    x = torch.tensor(g, device="cuda")
                    rest = [torch.empty_like(x) for _ in range(2)]
                    torch.cuda.synchronize()
                    assert lib().omni3d_adjoint(t.handle, x.data_ptr(), x.data_ptr(), *[r.data_ptr() for r in rest], 1) == 0
                    got = [r.cpu().numpy().reshape(dims[::-1]) for r in (x, *rest)]
                else:
                    got = t.adjoint(g)
                assert _copies(t) == 0
                for p, q in zip(got, want):
                    assert synthetic.relative_l2(p, q, gauge="none") < 1e-5
                _same(t.solve(*a, curl=curl), first, method)


def test_operator_that_fits_without_the_copies(omni):
    """Whether the anchor operator passes its automatic limit does not depend on the skewed copies: they
    go when it fits only without them.  40^3 voxels: copies of 176 bytes a voxel, at most half of the free memory."""
    dims = (40, 40, 40)
    f = synthetic.blobs(dims=dims, count=4, sigma_range=(3.0, 8.0), noise=0.05, seed=126)
    a = [f[k] for k in ("ax", "ay", "az")]
    memory = lib().omni3d_test_memory
    memory.restype, memory.argtypes = None, [C.c_void_p, C.c_longlong]

    def solve(nbytes):
        with omni.Omni3D(dims, f["spacing"], omni.icosphere(4), max_iter=5, gauge="mean") as s:
            if nbytes:
                memory(s.handle, nbytes)
            r = s.solve(*a)
            return r, _copies(s)

    want, copies = solve(0)
    assert copies == 1
    need = 10 * want.stats["n_links"]  # 80 % hold 8 bytes a link
    copied = 176 * 40**3
    assert 2 * 192 * 40**3 < need - need // 100  # skewed copies are taken in all three
    for nbytes, solver, skewed in ((need + copied // 2, 0, 0),  # the operator fits without the copies,
                                   (need + copied + 4096, 0, 1),  # beside them,
                                   (need - need // 100, 1, 1)):  # not at all
        r, copies = solve(nbytes)
        assert (r.stats["solver_used"], copies) == (solver, skewed)
        _same(r, want, "plain")
