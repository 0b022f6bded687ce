"""The QP norm estimates with a row that holds most of the matrix (estimated on the host) and with the same vector
length in short rows (on the device, 11 chunks of it and an entry more): the reference's number either way."""
import numpy as np
import pytest

from sih26_b200 import lpgen, pdhg
from tests.test_gpu_qp_norms import _estimate

pytestmark = pytest.mark.gpu


def _dense_row(n):
    lp = lpgen.qp_planted(1, n, 1, seed=6)
    assert lp.num_nonzeros == n
    return lp


@pytest.mark.parametrize("lp", [_dense_row(30_000), lpgen.qp_planted(3001, 12_001, 2, seed=6),
                                lpgen.qp_planted(30_000, 11, 20_000, seed=6)],
                         ids=["one dense row", "short rows", "dense columns"])
def test_the_references_number(lp):
    s = pdhg.solve_qp(lp, pdhg.Options(qp_assume_convex=True, iteration_limit=1))
    assert s.spectral_norm == _estimate(lp)
    assert np.isfinite(s.col_value).all()
