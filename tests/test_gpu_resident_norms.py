"""The FP32 level on a cluster whose shared memory does not hold the FP64 view that the norm estimate wants: the
estimate runs out of L2 (10,000 x 15,000 and 8,000 x 14,000: no FP64 plan) or streams both sides (6,000 x
12,000) or one (5,000 x 12,000). The answers are the grid-wide kernels' bit for bit, over the hand-over to the FP64
polish too, which takes a cluster's state to the grid-wide kernels."""
import numpy as np
import pytest

from sih26_b200 import lpgen
from sih26_b200 import pdhg as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,per_col", [(10_000, 15_000, 2), (8000, 14_000, 3), (6000, 12_000, 3), (5000, 12_000, 3)])
def test_the_grid_wide_kernels_bits(m, n, per_col):
    lp = lpgen.uniform_planted(m, n, per_col, seed=3)
    blocks = -(-(lp.num_nonzeros + m + n) // 4096)
    assert 2 <= blocks <= 16
    # the FP32 level is left at 1e-3 for the FP64 one, whose loop then runs to the limit
    kw = dict(pdhg_tolerance=1e-14, pdhg_stop_rule="relative_kkt", pdhg_precision="mixed", pdhg_algorithm="halpern",
              pdhg_mixed_switch_tolerance=1e-3, iteration_limit=3000)
    own = P.solve_pdhg(lp, P.Options(**kw))
    grid = P.solve_pdhg(lp, P.Options(pdhg_grid_blocks=blocks, **kw))
    assert own.spectral_norm == grid.spectral_norm
    assert 0 < own.fp32_iterations < own.iterations
    assert (own.status, own.iterations, own.fp32_iterations, own.restarts) == (
        grid.status, grid.iterations, grid.fp32_iterations, grid.restarts)
    for field in ("col_value", "row_dual", "col_dual"):
        assert np.array_equal(getattr(own, field), getattr(grid, field)), field
