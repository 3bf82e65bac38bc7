"""The bit-reproducible mode (params.deterministic) gives the bits of the inputs: not those of the
layout a context's free memory allowed, of the line order, or of a field solved before."""
import numpy as np
import pytest
from test_gpu_row_major import METHODS, _copies

from omni3d import synthetic

pytestmark = pytest.mark.gpu

DIMS = (29, 33, 26)


def _bits(a):
    return np.ascontiguousarray(np.asarray(a, np.float32)).view(np.uint32)


def _equal(a, b):
    np.testing.assert_array_equal(_bits(a.p), _bits(b.p))
    np.testing.assert_array_equal(_bits(a.count), _bits(b.count))


def _field(orc):
    f = synthetic.blobs(dims=DIMS, count=4, sigma_range=(2.0, 6.0), noise=0.10, seed=130, sphere_radius=4.0)
    curl = orc.curl(DIMS, f["spacing"], f["ax"], f["ay"], f["az"], f["mask"])
    return f, [f[k] for k in ("ax", "ay", "az")], curl, float(np.percentile(curl[curl > 0], 85))


@pytest.mark.parametrize("solver", ["anchor", "sweep"])
@pytest.mark.parametrize("method", METHODS)
def test_bits_do_not_depend_on_the_layout(omni, orc, method, solver):
    f, a, curl, thr = _field(orc)
    with omni.Omni3D(DIMS, f["spacing"], omni.icosphere(3), max_iter=5, method=method, threshold=thr, gauge="mean",
                     solver=solver, deterministic=True) as s:
        skewed = s.solve(*a, curl=curl)
        _copies(s, lose=True)
        row_major = s.solve(*a, curl=curl)
        assert _copies(s) == 0
    _equal(row_major, skewed)


@pytest.mark.parametrize("solver", ["anchor", "sweep"])
@pytest.mark.parametrize("method", METHODS)
def test_bits_do_not_depend_on_the_line_order(omni, orc, method, solver):
    f, a, curl, thr = _field(orc)
    runs = []
    for tile_width, dir_group in ((8, 32), (4, 1), (16, 5)):
        with omni.Omni3D(DIMS, f["spacing"], omni.icosphere(3), max_iter=5, method=method, threshold=thr, gauge="mean",
                         solver=solver, deterministic=True, tile_width=tile_width, dir_group=dir_group) as s:
            runs.append(s.solve(*a, curl=curl))
    for r in runs[1:]:
        _equal(r, runs[0])


def test_bits_do_not_depend_on_the_field_before(omni):
    """The captured iterations hold the bounds of the sums they were captured for.  Minimum-curl paths
    follow the field: here up to 943 lines cross a voxel in the first field and 7305 in the second.
    One least curl far below the others makes the sums' resolution, which follows from the bounds,
    coarse enough to show in the bits."""
    dims = (20, 18, 16)
    rng = np.random.default_rng(131)
    k, j, i = np.meshgrid(*[np.arange(n) for n in dims[::-1]], indexing="ij")
    spread = rng.uniform(1.0, 2.0, i.shape)
    centred = 1.0 + 0.01 * ((i - 10) ** 2 + (j - 9) ** 2 + (k - 8) ** 2)
    a = [rng.normal(size=i.size).astype(np.float32) for _ in range(3)]
    fields = []
    for c in (spread, centred):
        c[8, 9, 10] = 1e-9
        fields.append(c.astype(np.float32).reshape(-1))
    opts = dict(max_iter=40, tol=1e-30, method="weighted_mini_curl", gauge="mean", deterministic=True)
    with omni.Omni3D(dims, 1.0, omni.icosphere(3), **opts) as s:
        s.solve(*a, curl=fields[0])
        after = s.solve(*a, curl=fields[1])
    with omni.Omni3D(dims, 1.0, omni.icosphere(3), **opts) as s:
        alone = s.solve(*a, curl=fields[1])
    assert after.stats["iterations"] == alone.stats["iterations"] == 40
    _equal(after, alone)
