"""Restarts of the FP32 level on a cluster of several blocks (resident.cuh), Halpern operator.

A restart refills every block's copy of x, and the next step's new entries come from the other blocks into the
same buffer: with a refill that is not ordered before those stores a block keeps a zero where its peers have
the new entry, and the answer changes from run to run. The same LP many times over, with restarts enough, is the
grid-wide kernels' answer every time, bit for bit."""
import numpy as np
import pytest

from sih26_b200 import lpgen
from sih26_b200 import pdhg as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,per_col", [(300, 700, 9), (1000, 2500, 10), (2000, 5000, 10), (1999, 5403, 10)])
def test_answers_do_not_change_from_run_to_run(m, n, per_col):
    lp = lpgen.uniform_planted(m, n, per_col, seed=11)
    work = lp.num_nonzeros + m + n
    blocks = -(-work // 4096)
    assert 2 <= blocks <= 16
    kw = dict(pdhg_tolerance=1e-9, pdhg_stop_rule="relative_kkt", pdhg_precision="mixed",
              pdhg_algorithm="halpern", iteration_limit=3000, pdhg_mixed_switch_tolerance=1e-12)
    grid = P.solve_pdhg(lp, P.Options(pdhg_grid_blocks=blocks, **kw))
    assert grid.restarts >= 3
    for _ in range(25):
        own = P.solve_pdhg(lp, P.Options(**kw))
        assert (own.iterations, own.restarts, own.evaluations) == (grid.iterations, grid.restarts, grid.evaluations)
        for field in ("col_value", "row_dual", "col_dual"):
            assert np.array_equal(getattr(own, field), getattr(grid, field)), field
