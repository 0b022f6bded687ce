"""Batched LPs with rows and columns beyond a segment of 512 entries whose vectors pass through shared memory in
turns or are gathered out of L2: the single-LP path's answer to rounding, as for the batch's other ways."""
import numpy as np
import pytest
import scipy.sparse as sp

from sih26_b200 import pdhg as P
from sih26_b200.lpgen import LP

pytestmark = pytest.mark.gpu


def _lp(m, n, lengths, transpose=False):
    """Rows of the given lengths on top of three entries a column (row-wise where transposed)."""
    rng = np.random.default_rng(m + n)
    rows, cols = [], []
    for i, length in enumerate(lengths):
        rows.append(np.full(length, i))
        cols.append(rng.choice(n, length, replace=False))
    rows.append(rng.integers(0, m, 3 * n))
    cols.append(np.repeat(np.arange(n), 3))
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    a = sp.csc_matrix((rng.standard_normal(len(rows)), (rows, cols)), shape=(m, n))
    if transpose:
        a = sp.csc_matrix(a.T)
    a.sum_duplicates()
    a.sort_indices()
    m, n = a.shape
    act = a @ rng.uniform(0, 1, n)
    return LP(num_rows=m, num_cols=n, col_starts=a.indptr.astype(np.int32), row_indices=a.indices.astype(np.int32),
              values=a.data, cost=rng.standard_normal(n), col_lower=np.zeros(n), col_upper=np.full(n, 2.0),
              row_lower=act, row_upper=act)


@pytest.mark.parametrize("algorithm", ["halpern", "reference"])
@pytest.mark.parametrize("m,n,lengths,transpose", [
    (40, 20_011, [513, 1024, 1025, 20_011], False),   # in turns; a segment and one, two full, two and one, all
    (9000, 20_011, [20_011, 511, 512], False),        # beside short rows
    (40, 20_011, [513, 20_011], True),                # long columns
    (1, 5000, [5000], False),                         # one block
    (300, 30_011, [30_011, 600], False),              # out of L2
])
def test_the_single_lp_paths_answer(m, n, lengths, transpose, algorithm):
    lp = _lp(m, n, lengths, transpose)
    opts = P.Options(pdhg_tolerance=1e-14, pdhg_stop_rule="relative_kkt", pdhg_algorithm=algorithm,
                     iteration_limit=120 if algorithm == "halpern" else 60)
    one, got = P.solve_pdhg(lp, opts), P.batch_solve([lp], opts)[0]
    assert (got.status, got.iterations, got.restarts) == (one.status, one.iterations, one.restarts)
    for field in ("col_value", "row_dual", "col_dual"):
        a, b = getattr(got, field), getattr(one, field)
        assert np.linalg.norm(a - b) <= 1e-9 * max(1.0, np.linalg.norm(b)), field
