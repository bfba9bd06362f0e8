"""Fixed iteration counts of 1D grids in calls of any length: a few iterations
run one per launch, more in one launch, with the iterates of one long call, also
between steps and before the iterations that itmax leaves after a step's last
check."""
import numpy as np
import pytest

import ptdiff
from ptdiff import scripts as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["diff_1D_lin", "diff_1D_linstep", "diff_1D_nonlin"])
@pytest.mark.parametrize("n", [3, 40, 333, 8192, 8193])
def test_calls_of_any_length(name, n):
    s = S.SCRIPTS[name]
    H0, D = S.initial_condition(s, n), S.step_field(s, n) if s.model == S.LINSTEP else None
    out = []
    for calls in ([1, 1, 2, 5, 1, 6, 3, 20, 1], [40], [2] * 20):
        with ptdiff.Solver(ptdiff.make_params(s, (n,))) as sol:
            sol.set_state(H0, D)
            for k in calls:
                sol.iterate(k)
            assert sol.counters()[1] == 40
            out.append(sol.get_state())
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])


@pytest.mark.parametrize("n", [333, 9000])
@pytest.mark.parametrize("itmax", [21, 24, 29])
def test_iterations_between_steps_and_after_the_last_check(n, itmax):
    s = S.SCRIPTS["diff_1D_nonlin"]
    out = []
    for resid in ("mixed", "consistent"):   # the second: one launch per iteration throughout
        with ptdiff.Solver(ptdiff.make_params(s, (n,), itmax=itmax, tol=1e-300, resid=resid)) as sol:
            sol.set_state(S.initial_condition(s, n))
            for k in (1, 3):
                assert list(sol.step(2)[0]) == [itmax] * 2
                sol.iterate(k)
            out.append(sol.get_state())
    assert np.array_equal(out[0], out[1])
