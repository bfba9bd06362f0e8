"""Waits of the one-launch steps that run out: the kernel gives up and returns,
the calls report it, and a new state makes the context good again; and check
blocks too long for a wait's limit, which run one iteration per launch."""
import numpy as np
import pytest

import ptdiff
from ptdiff import _abi
from ptdiff import scripts as S

pytestmark = pytest.mark.gpu

CASES = [("diff_2D_nonlin", (128, 96)), ("diff_2D_linstep", (300, 210)), ("diff_3D_nonlin_multixpu", (40, 36, 33))]


def fields(s, shape):
    return S.initial_condition(s, *shape), S.step_field(s, *shape) if s.model == S.LINSTEP else None


def timed_out(call, *a):
    with pytest.raises(_abi.PtdError) as e:
        call(*a)
    assert e.value.status == _abi.PTD_ETIMEOUT


@pytest.mark.parametrize("checks", [True, False])
@pytest.mark.parametrize("name,shape", CASES)
def test_a_wait_that_gives_up(name, shape, checks):
    s = S.SCRIPTS[name]
    H0, D = fields(s, shape)
    p = ptdiff.make_params(s, shape)
    with ptdiff.Solver(p) as sol:
        sol.set_state(H0, D)
        want_its = list(sol.step(2)[0])
        want = sol.get_state()
    with ptdiff.Solver(p) as sol:
        sol.set_state(H0, D)
        sol.step(1)
        sol.set_wait_limit(1)   # an edge takes more polls than one to arrive
        if checks:
            timed_out(sol.step, 1)
        else:
            sol.iterate(200)
            timed_out(sol.sync)
        timed_out(sol.get_state)
        timed_out(sol.step, 1)
        timed_out(sol.iterate, 5)
        timed_out(lambda: sol.set_launch_config(warps2d=2, chunk2d=8))
        sol.set_wait_limit(0)
        timed_out(sol.step, 1)
        sol.set_state(H0, D)
        assert list(sol.step(2)[0]) == want_its and np.array_equal(sol.get_state(), want)


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
