"""Memory that the library keeps between calls is given back on request: what a solve leaves is freed by the
first release, a second has nothing to free, and the next solve's answer is the same."""
import numpy as np
import pytest

from sih26_b200 import lpgen
from sih26_b200 import pdhg as P

pytestmark = pytest.mark.gpu


def test_release_gives_the_memory_back():
    lp = lpgen.uniform_planted(60, 150, 4, seed=2)
    before = P.solve_pdhg(lp, P.Options())
    assert P.release_memory() >= 64 << 20  # a solve's first chunk
    assert P.release_memory() == 0
    after = P.solve_pdhg(lp, P.Options())
    assert np.array_equal(before.col_value, after.col_value)
    with pytest.raises(P.GpuError):
        P.release_memory(10_000)
