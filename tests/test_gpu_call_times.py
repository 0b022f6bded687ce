"""What a call reports of its own time, on an LP that one cluster solves in one launch: the norm estimate belongs
to the set-up and the report to neither, the timed iteration launches hold the iterations alone, and the verbose
line names the norm.

An LP stopped at its first iteration has a loop of nothing: some 10 us of launch, entry and copy are left of the
150 us and more that the norm estimate and the report take beside them; 100 us leave room for the host."""
import numpy as np
import pytest

from sih26_b200 import lpgen
from sih26_b200 import pdhg as P

pytestmark = pytest.mark.gpu


def _lp():
    return lpgen.uniform_planted(2000, 5000, 10, seed=3)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_sections(precision):
    lp = _lp()
    kw = dict(pdhg_tolerance=1e-12, pdhg_stop_rule="relative_kkt", pdhg_precision=precision,
              pdhg_algorithm="halpern", pdhg_profile_kernels=True, pdhg_mixed_stall_checks=-1)
    P.solve_pdhg(lp, P.Options(iteration_limit=40, **kw))
    none = [P.solve_pdhg(lp, P.Options(iteration_limit=0, **kw)) for _ in range(7)]
    assert min(s.iterate_kernel_seconds for s in none) < 25e-6
    assert min(s.device_seconds for s in none) < 100e-6
    some = P.solve_pdhg(lp, P.Options(iteration_limit=400, **kw))
    assert some.iterations == 400
    # 400 iterations and 10 evaluations; an iteration takes 3 us at the least
    assert 400 * 3e-6 < some.iterate_kernel_seconds < some.device_seconds
    for s in (*none, some):
        assert s.setup_seconds > 0.0
        assert s.setup_seconds + s.device_seconds < s.solve_seconds


def test_the_verbose_line_names_the_norm(capfd):
    lp = _lp()
    kw = dict(pdhg_tolerance=1e-6, pdhg_stop_rule="relative_kkt", pdhg_algorithm="halpern", iteration_limit=330)
    quiet = P.solve_pdhg(lp, P.Options(**kw))
    capfd.readouterr()
    loud = P.solve_pdhg(lp, P.Options(log_to_console=True, **kw))
    assert f"||A||_2 ~ {loud.spectral_norm:.4e}" in capfd.readouterr().out
    assert (loud.iterations, loud.spectral_norm) == (quiet.iterations, quiet.spectral_norm)
    assert np.array_equal(loud.col_value, quiet.col_value)
