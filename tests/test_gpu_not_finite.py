"""Tolerance-driven solves whose pressures leave FP32's range: a change that is not finite does not meet
the tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gauge,ref", [("none", 0), ("point", -1), ("point", 1)])
def test_infinite_change_is_not_convergence(omni, gauge, ref):
    """One direction, an entry that its own line alone crosses and an initial pressure of 3e38 there:
    the first iteration adds it to itself (numer = p + p_init, count 1), which is infinite.  The
    reference pressure of the point gauge is below or above zero."""
    dims = (9, 8, 7)
    dirs = omni.icosphere(2)[5:6]
    zero = np.zeros(int(np.prod(dims)), np.float32)
    with omni.Omni3D(dims, 1.0, dirs, max_iter=1) as s:
        count = s.solve(zero, zero, zero).count.reshape(-1)
        entries = np.unique(s.line_table()[:, 0])
    alone = entries[count[entries] == 1]
    p0 = zero.copy()
    p0[alone[0]] = 3e38
    at = int(alone[-1])
    p0[at] = ref
    c = dict(gauge=gauge, ref=(at % 9, at // 9 % 8, at // 72))
    with omni.Omni3D(dims, 1.0, dirs, max_iter=6, tol=1e-3, **c) as s:
        r = s.solve(zero, zero, zero, p_init=p0.reshape(dims[::-1]))
    # the second iteration's row sums are NaN, which ends the iterations
    assert r.stats["iterations"] == 3
