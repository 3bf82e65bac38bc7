"""The line-order tuning (params.autotune) times the walks that the context will run."""
import ctypes as C

import numpy as np
import pytest
from test_gpu_parity import TOL_P_PLAIN
from test_gpu_row_major import _copies

from omni3d import synthetic

pytestmark = pytest.mark.gpu


def test_tuning_times_the_contexts_layout(omni):
    """Skewed copies at this size.  They are given back: a tuned context solves like an untuned one, and
    row-major where its first field finds no memory for them."""
    tuned = omni.lib().omni3d_test_tuned
    tuned.restype, tuned.argtypes = C.c_int, [C.c_void_p]
    dims = (37, 33, 35)
    f = synthetic.blobs(dims=dims, count=3, sigma_range=(2.0, 5.0), noise=0.05, seed=140)
    runs = []
    for tune, lose in ((False, False), (True, False), (True, True), (True, False)):
        with omni.Omni3D(dims, f["spacing"], omni.icosphere(3), max_iter=4, autotune=tune) as s:
            assert tuned(s.handle) == (1 if tune else -1)
            assert _copies(s, lose=lose) == 0  # chosen at the first field
            runs.append(s.solve(f["ax"], f["ay"], f["az"]))
            assert _copies(s) == int(not lose)
    for r in runs[1:]:
        np.testing.assert_array_equal(r.count, runs[0].count)
        assert synthetic.relative_l2(r.p, runs[0].p) < 2 * TOL_P_PLAIN
