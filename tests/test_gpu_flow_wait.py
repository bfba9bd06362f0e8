"""Check blocks too long for a wait's limit run one iteration per launch: the
one-launch step's judge waits for a whole block."""
import pytest

import ptdiff
from ptdiff import scripts as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,shape,nchk,one_launch", [("diff_2D_nonlin", (33, 31), 1 << 18, True),
                                                        ("diff_3D_lin_multixpu", (33, 32, 32), 1 << 18, True),
                                                        ("diff_2D_nonlin", (33, 31), (1 << 18) + 1, False)])
def test_check_blocks_longer_than_a_wait_lasts(name, shape, nchk, one_launch):
    s = S.SCRIPTS[name]
    with ptdiff.Solver(ptdiff.make_params(s, shape, nchk=nchk, itmax=nchk)) as sol:
        sol.set_state(S.initial_condition(s, *shape))
        before = sol.counters()[0]
        iters, _ = sol.step(1)
        launches = sol.counters()[0] - before
    assert list(iters) == [nchk]
    assert (launches == 1) if one_launch else (launches > nchk)
