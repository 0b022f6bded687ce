"""Batched LPs whose vectors outgrow a block's shared memory, gathered out of L2 by clusters in a launch of their
own: the single-LP path's answer to rounding, and the same bits alone, beside LPs of the other classes, with one
cluster for all, and when the LP pauses between launches.

The tolerance is that of the batch's other ways to hold an LP: both run the same FP64 iteration, only the order of
sums differs, by a few roundings of 2^-53 in each of 120 steps of an operator that does not expand distances."""
import numpy as np
import pytest

from sih26_b200 import lpgen
from sih26_b200 import pdhg as P

pytestmark = pytest.mark.gpu

WHOLE = 212 * 1024 // 8  # FP64 entries of a vector that fits alone


def _options(algorithm):
    return P.Options(pdhg_tolerance=1e-14, pdhg_stop_rule="relative_kkt", pdhg_algorithm=algorithm,
                     iteration_limit=120 if algorithm == "halpern" else 60)


@pytest.mark.parametrize("algorithm", ["halpern", "reference"])
@pytest.mark.parametrize("m,n,per_col", [(9000, WHOLE + 1, 2), (WHOLE + 1, 9001, 6), (40001, 100003, 3)])
def test_alone_and_in_the_mix(m, n, per_col, algorithm):
    lp = lpgen.uniform_planted(m, n, per_col, seed=1)
    opts = _options(algorithm)
    one = P.solve_pdhg(lp, opts)
    alone = P.batch_solve([lp], opts)[0]
    assert (alone.status, alone.iterations, alone.restarts) == (one.status, one.iterations, one.restarts)
    for field in ("col_value", "row_dual", "col_dual"):
        a, b = getattr(alone, field), getattr(one, field)
        assert np.linalg.norm(a - b) <= 1e-9 * max(1.0, np.linalg.norm(b)), field
    others = [lpgen.uniform_planted(50, 120, 4, seed=9), lpgen.uniform_planted(800, 2003, 9, seed=1),
              lpgen.uniform_planted(9001, 20001, 8, seed=1)]
    others_alone = [P.batch_solve([o], opts)[0] for o in others]
    for config in (dict(chunk_attempts=0), dict(chunk_attempts=40, clusters=1), dict(chunk_attempts=40)):
        with P.Server(pool_bytes=1 << 29, **config) as srv:
            got = srv.solve_all([lp, *others, lp], opts)
        for s, want in zip(got, [alone, *others_alone, alone]):
            assert s.iterations == want.iterations
            assert np.array_equal(s.col_value, want.col_value)


def test_few_entries_in_long_vectors_on_one_block():
    lp = lpgen.uniform_planted(40_000, 12_000, 1, seed=1)  # 12,000 nonzeros: one block
    opts = _options("halpern")
    one, got = P.solve_pdhg(lp, opts), P.batch_solve([lp], opts)[0]
    assert (got.status, got.iterations) == (one.status, one.iterations)
    assert np.linalg.norm(got.col_value - one.col_value) <= 1e-9 * max(1.0, np.linalg.norm(one.col_value))
