"""A column's reduced cost is summed from its cost on, entry by entry (pdhg.cpp:172-199), on every path of the
residual check: with cost 1e16 and terms -1e16 and 1 it is exactly 1, and 0 if the terms are summed first."""
import ctypes as C

import numpy as np
import pytest

from sih26_b200.lpgen import LP
from tests.test_zz_no_alloc import _call, _device_problem, _lib

pytestmark = pytest.mark.gpu


def _lp(n):
    """Column 0 holds the two entries, the others are empty and fixed at zero cost."""
    inf = np.inf
    starts = np.full(n + 1, 2, np.int32)
    starts[0] = 0
    cost = np.zeros(n)
    cost[0] = 1e16
    lower, upper = np.zeros(n), np.zeros(n)
    lower[0], upper[0] = -inf, inf
    return LP(num_rows=2, num_cols=n, col_starts=starts, row_indices=np.array([0, 1], np.int32), values=np.ones(2),
              cost=cost, col_lower=lower, col_upper=upper, row_lower=np.zeros(2), row_upper=np.zeros(2))


@pytest.mark.parametrize("n,out_of_order", [(1, False), (40, False), (8000, False), (8000, True)])
def test_the_cost_comes_first(n, out_of_order):
    torch = pytest.importorskip("torch")
    lp = _lp(n)
    keep = []
    prob = _device_problem(lp, torch, keep)
    if out_of_order:  # column 2 would begin before column 1 ends: each lane then reads its own column
        starts = np.array(lp.col_starts)
        starts[1], starts[2] = 2, 0
        starts[3:] = 0
        bad = torch.as_tensor(starts, device="cuda:0")
        keep.append(bad)
        prob.col_starts = C.cast(bad.data_ptr(), C.POINTER(C.c_int32))
    got = _call(_lib(), torch, prob, np.zeros(n), np.array([1e16, -1.0]), torch.cuda.Stream())
    # the free column's reduced cost is the only dual violation
    assert got["absolute_dual"] == 1.0
