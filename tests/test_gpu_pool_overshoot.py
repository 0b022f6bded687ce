"""LPs whose region outgrows the server's pool take device memory beside it one at a time: each runs in a launch
that no other such LP shares, LPs that fit the pool run beside them, and the answers are those of a large pool."""
import numpy as np
import pytest

from sih26_b200 import lpgen
from sih26_b200 import pdhg as P

pytestmark = pytest.mark.gpu


def test_one_at_a_time():
    big = [lpgen.uniform_planted(2000, 5000, 10, seed=k) for k in range(4)]
    small = lpgen.uniform_planted(60, 150, 4, seed=1)
    opts = P.Options(pdhg_tolerance=1e-6, pdhg_stop_rule="relative_kkt", pdhg_algorithm="halpern")
    with P.Server(chunk_attempts=0) as srv:
        want = srv.solve_all([small, *big], opts)
        assert srv.stats()["rounds"] == 1
    # what both copies of the matrix, the vectors and the lists take, with little to spare
    with P.Server(chunk_attempts=0, pool_bytes=24 * big[0].num_nonzeros + 136 * 7000 + (96 << 10)) as srv:
        got = srv.solve_all([small, *big], opts)
        assert srv.stats()["rounds"] == 4
    for g, w in zip(got, want):
        assert (g.status, g.iterations) == (w.status, w.iterations)
        assert np.array_equal(g.col_value, w.col_value)
