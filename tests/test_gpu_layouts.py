"""The GPU path at the sizes where its layouts and its choices of kernel change: volumes of two
to a few cells a side and around the 32-wide tiles (the walks' skewed copies, whose planes wrap
at the y extent), operators around the link kinds' limits (vector in shared memory, one panel of
columns, two, 32-bit links), grids around the filtered walk's limit.  The references are the
FP64 oracle, the oracle's lines and staircases, and the sweep solver, which uses no operator."""
import numpy as np
import pytest
from test_gpu_parity import TOL_P_PLAIN, TOL_PN, _lines_oracle

from omni3d import synthetic

pytestmark = pytest.mark.gpu

MODES = {"plain": 0, "select": 1, "weighted": 2}


def _random_field(dims, seed, scale=1.0):
    rng = np.random.default_rng(seed)
    return [(scale * rng.normal(size=int(np.prod(dims)))).astype(np.float32) for _ in range(3)]


@pytest.mark.parametrize("method", ["plain", "select", "weighted"])
@pytest.mark.parametrize("dims", [(2, 3, 5), (5, 2, 3), (31, 33, 32), (65, 5, 7), (4, 64, 33), (33, 3, 66)])
def test_sweep_over_skewed_copies(omni, orc, dims, method):
    """One sweep of every method against the FP64 oracle, at the bar of the sweep parity test."""
    h = (1e-3, 1e-3, 1e-3)
    dirs = omni.icosphere(3)
    a = _random_field(dims, 100)
    p = np.random.default_rng(101).normal(size=int(np.prod(dims))).astype(np.float32)
    curl, thr = None, 0.0
    if method != "plain":
        curl = orc.curl(dims, h, *a, np.ones(int(np.prod(dims)), np.float32))
        thr = float(np.percentile(curl, 80)) if method == "select" else 0.0
    epn, ecnt = orc.sweep(dims, h, dirs, *a, p, mode=MODES[method], thr=thr, curl=curl, precision="f64", nthreads=4)
    with omni.Omni3D(dims, h, dirs, max_iter=2, method=method, threshold=thr) as s:
        for call in range(2):  # the second after a solve, when a plain sweep's counts are known
            pn, cnt = s.sweep(*a, p, curl=curl)
            assert synthetic.relative_l2(pn.reshape(-1), epn, gauge="none") < TOL_PN
            if method == "plain":
                np.testing.assert_array_equal(cnt.reshape(-1), ecnt.astype(np.float32))
            else:
                assert synthetic.relative_l2(cnt.reshape(-1), ecnt, gauge="none") < TOL_PN
            s.solve(*a, curl=curl)


# 6 N^2 - 12 N + 8 anchors: 16226 and 16856 around the shared-memory vector's least size, 54152 and
# 55298 around one panel, 109352 and 110978 around two
@pytest.mark.parametrize("n", [53, 54, 96, 97, 136, 137])
@pytest.mark.parametrize("option", ["", "sweep_fp64", "deterministic"])
def test_plain_operator_kinds(omni, n, option):
    """The anchor solver against the sweep solver: the same iterates up to the order of sums,
    each within TOL_P_PLAIN of the FP64 ones."""
    dims = (n, n, n)
    f = synthetic.blobs(dims=dims, count=4, sigma_range=(3.0, 9.0), noise=0.05, seed=102)
    dirs = omni.icosphere(2)
    out = []
    for solver, tol in (("sweep", 0.0), ("anchor", 0.0), ("anchor", 1e-30)):
        with omni.Omni3D(dims, f["spacing"], dirs, max_iter=5, solver=solver, tol=tol, gauge="mean",
                         **({option: True} if option else {})) as s:
            out.append(s.solve(f["ax"], f["ay"], f["az"]))
    assert out[1].stats["solver_used"] != out[0].stats["solver_used"]
    for r in out[1:]:
        assert synthetic.relative_l2(r.p, out[0].p) < 2 * TOL_P_PLAIN
        np.testing.assert_array_equal(r.count, out[0].count)


@pytest.mark.parametrize("dims", [(9, 34, 5), (54, 54, 54), (97, 97, 97)])
def test_plain_adjoint_is_the_transpose(omni, dims):
    """<g, J h> = <J^T g, h> at h = J^T g, where the left side is |J^T g|^2 and nothing cancels:
    p's error is below TOL_P_PLAIN of it, and g and J h are far from orthogonal."""
    dirs = omni.icosphere(2)
    a = _random_field(dims, 103)
    g = np.random.default_rng(104).normal(size=int(np.prod(dims))).astype(np.float32)
    with omni.Omni3D(dims, 1.0, dirs, max_iter=6, gauge="none") as s:
        p0 = s.solve(*a).p.reshape(-1).astype(np.float64)
        gt = [np.asarray(x).reshape(-1) for x in s.adjoint(g)]
        size = 50.0 / max(float(np.abs(x).max()) for x in gt)
        h = [(size * x).astype(np.float32) for x in gt]
        p1 = s.solve(*[x + y for x, y in zip(a, h)]).p.reshape(-1).astype(np.float64)
    lhs = float(np.dot(g, p1 - p0))
    rhs = float(sum(np.dot(x.astype(np.float64), y) for x, y in zip(gt, h)))
    assert abs(lhs - rhs) <= 1e-4 * abs(lhs)


# (below about 1e-19 the curl's squares underflow, and a selected solve has no anchor to start from)
@pytest.mark.parametrize("method,scale", [("plain", 1e-25), ("plain", 1.0), ("plain", 1e15), ("select", 1e-15),
                                          ("select", 1.0), ("select", 1e15)])
def test_fixed_point_scales(omni, method, scale):
    """The bit-reproducible mode's terms are scaled in FP32 by two factors: over magnitudes that
    need either, it agrees with the default mode to that mode's FP32 rounding."""
    dims = (20, 17, 23)
    a = _random_field(dims, 105, scale)
    dirs = omni.icosphere(2)
    r = []
    for det in (True, False):
        with omni.Omni3D(dims, 1.0, dirs, max_iter=4, method=method, threshold=1e30, gauge="mean", deterministic=det) as s:
            r.append(s.solve(*a).p.astype(np.float64) / scale)
    assert synthetic.relative_l2(r[0], r[1]) < 1e-5


@pytest.mark.parametrize("dims,level,ndir", [((40, 36, 44), 2, 42), ((3, 2, 90), 3, 162), ((2048, 3, 2), 1, 3),
                                             ((2, 2049, 3), 1, 3)])
def test_walks_and_misses_bit_exact(omni, orc, match_lines, dims, level, ndir):
    """The filtered walks (up to 2048 cells a side) and the lines left out beforehand: the oracle's
    line table and staircases."""
    dirs = omni.icosphere(level)[:ndir]
    with omni.Omni3D(dims, 1e-3, dirs, max_iter=1) as s:
        got = s.line_table().astype(np.int64)
        got[:, 0] &= 0xFFFFFFFF
        got[:, 1] &= 0xFFFFFFFF
        exp, geo = _lines_oracle(orc, dims, 1.0, dirs)
        at = match_lines(got, exp)
        for k in range(0, len(exp), max(1, len(exp) // 400)):
            io, xyz = geo[k]
            ax = orc.walk(dims, io, xyz, dirs[exp[k, 2]])
            assert any(np.array_equal(s.line_steps(i), ax) for i in at[k]), k
