"""A Hessian whose factorisation overflows: inf - inf makes a pivot that is neither below nor within the slack,
and check_convexity (src/qp/convexity.cpp:30-134) goes on with it, so that every later pivot is no number either
and the Hessian passes. The device's panels pass it on to the rows below them alike."""
import numpy as np
import pytest

from sih26_b200 import pdhg as P
from tests.test_gpu_convexity import _qp

pytestmark = pytest.mark.gpu


def _hessian(n, i, bad):
    q = np.eye(n)
    for c, big in ((0, 1e305), (1, -1e305)):  # l_i0 l_20 = inf and l_i1 l_21 = -inf
        q[2, c] = q[c, 2] = 1e4
        q[i, c] = q[c, i] = big
    q[2, 2] = 1e9
    q[bad, bad - 1] = q[bad - 1, bad] = 2.0  # a pivot of -3 by itself
    return q


def _reference(q):
    """The loop of check_convexity; the first column that it rejects, or None."""
    n = len(q)
    slack = 1e-10 * max(1.0, np.abs(np.diag(q)).max())
    l, d = np.zeros((n, n)), np.zeros(n)
    with np.errstate(all="ignore"):
        for j in range(n):
            pivot = q[j, j]
            for k in range(j):
                pivot -= l[j, k] * l[j, k] * d[k]
            if pivot < -slack:
                return j
            if pivot <= slack:
                continue
            d[j] = pivot
            below = q[j + 1:, j].copy()
            for k in range(j):
                below -= l[j + 1:, k] * l[j, k] * d[k]
            l[j + 1:, j] = below / pivot
    return None


@pytest.mark.parametrize("i", [3, 31, 32, 40])
def test_the_verdict_is_the_references(i):
    n, bad = 128, 100
    q = _hessian(n, i, bad)
    assert _reference(q) is None
    p = q.copy()
    p[i, :2] = p[:2, i] = 0.0
    assert _reference(p) == bad
    opts = P.Options(qp_tolerance=1e-6, iteration_limit=1)
    assert f"column {bad}" in P.solve_qp(_qp(n, p), opts).message
    try:
        s = P.solve_qp(_qp(n, q), opts)
    except P.GpuError as e:  # past the test, the steps of a Hessian of 1e305 are no numbers
        assert "not finite" in str(e)
    else:
        assert s.status != "model_error"
