"""Batched LPs without rows or without columns, of sizes that fit a block's shared memory, that do not, and of
several windows: the bound-only LP's optimum is each cost's cheaper bound (to the gap of the stopping
rule), and the LP without columns has nothing to move."""
import numpy as np
import pytest

from sih26_b200 import pdhg as P
from sih26_b200.lpgen import LP

pytestmark = pytest.mark.gpu

WINDOW = 212 * 1024 // 8


def _lp(m, n, seed=5):
    rng = np.random.default_rng(seed)
    none = np.zeros(0)
    return LP(num_rows=m, num_cols=n, col_starts=np.zeros(n + 1, np.int32), row_indices=np.zeros(0, np.int32),
              values=none, cost=rng.choice([-1.0, 1.0], n) * rng.uniform(0.5, 2.0, n), col_lower=-rng.uniform(1, 2, n),
              col_upper=rng.uniform(1, 2, n), row_lower=-rng.uniform(0, 1, m), row_upper=rng.uniform(0, 1, m))


@pytest.mark.parametrize("algorithm", ["halpern", "reference"])
@pytest.mark.parametrize("m,n", [(0, 40), (40, 0), (0, 6000), (6000, 0), (0, 2 * WINDOW + 5), (2 * WINDOW + 5, 0)])
def test_bounds_alone(m, n, algorithm):
    lp = _lp(m, n)
    opts = P.Options(pdhg_tolerance=1e-8, pdhg_stop_rule="relative_kkt", pdhg_algorithm=algorithm,
                     iteration_limit=2000)
    best = float(np.abs(np.where(lp.cost > 0, lp.cost * lp.col_lower, lp.cost * lp.col_upper)).sum())
    for got in [P.solve_pdhg(lp, opts), *P.batch_solve([lp, _lp(50, 120), lp], opts)[::2]]:
        assert got.status == "optimal"
        x = got.col_value
        assert np.all(x >= lp.col_lower) and np.all(x <= lp.col_upper)
        # a relative gap of 1e-8 of 1 + |primal| + |dual|, both within 1e-8 of the optimum
        assert abs(float(lp.cost @ x) + best) <= 1.01e-8 * (1 + 2 * best)
        assert np.array_equal(got.row_dual, np.zeros(m))
