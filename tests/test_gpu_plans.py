"""Plans that other tests do not reach: the 6-row LIN tile of the 2D one-launch
step, the 1D one-launch step of D = exp(m) H^3, and the marches that FP64 grids
take by default where no one-launch step serves them.  Each against the kernel
of one iteration per launch with another launch shape, bit for bit, in steps
that itmax stops."""
import numpy as np
import pytest

import ptdiff
from ptdiff import scripts as S

pytestmark = pytest.mark.gpu

EXPM = S.SCRIPTS["diff_1D_nonlin"].with_(name="expm", model=S.NONLIN_EXPM, shift=1.0, dirichlet=1.0, ic="linrange")


def fields(s, shape):
    D = None
    if s.model == S.LINSTEP:
        D = S.step_field(s, *shape)
    elif s.model == S.NONLIN_EXPM:
        D = S.log_coefficient_field(shape, seed=1)
    return S.initial_condition(s, *shape), D


def run(s, shape, cfg=None, iterate=0, steps=2, **kw):
    """H and the launches of two steps, or of `iterate` iterations."""
    H0, D = fields(s, shape)
    with ptdiff.Solver(ptdiff.make_params(s, shape, tol=1e-300, **kw)) as sol:
        if cfg:
            sol.set_launch_config(**cfg)
        sol.set_state(H0, D)
        before = sol.counters()
        if iterate:
            sol.iterate(iterate)
        else:
            iters, _ = sol.step(steps)
            assert list(iters) == [kw["itmax"]] * steps
        after = sol.counters()
        return sol.get_state(), after[0] - before[0], after[1] - before[1]


# 6 rows where 5 do not fit 151 SMs of 20 tiles: rows of tiles full and cut, a
# last column of one cell, and the largest; then the first grid that does not fit
@pytest.mark.parametrize("shape,one_launch", [((760, 680), True), ((745, 700), True), ((747, 700), True), ((684, 761), True),
                                              ((777, 720), True), ((777, 735), False)])
def test_lin_tile_of_six_rows(shape, one_launch):
    s, kw = S.SCRIPTS["diff_2D_lin"], {"itmax": 60, "nchk": 20}
    a = run(s, shape, **kw)
    b = run(s, shape, {"warps2d": 2, "chunk2d": 8}, **kw)
    assert np.array_equal(a[0], b[0])
    assert (a[1] <= 2) == one_launch and b[1] > 120


@pytest.mark.parametrize("n", [12, 13, 333, 1409, 9000])
def test_line_step_of_the_exponential_model(n):
    """The consistent residual runs one launch per iteration: the same iterates."""
    a = run(EXPM, (n,), steps=1, itmax=57, nchk=10)
    b = run(EXPM, (n,), iterate=57, resid="consistent")
    assert a[1] <= 2 < b[1]
    assert np.array_equal(a[0], b[0])


@pytest.mark.parametrize("name,shape,resid", [
    ("diff_2D_nonlin", (33, 34), "consistent"), ("diff_2D_linstep", (260, 251), "consistent"),
    ("diff_2D_lin", (95, 700), "consistent"), ("diff_2D_nonlin", (900, 811), "mixed"), ("diff_2D_lin", (1030, 725), "mixed"),
    ("diff_2D_linstep", (3000, 171), "mixed"), ("diff_3D_linstep_multixpu", (32, 23, 66), "consistent"),
    ("diff_3D_nonlin_multixpu", (90, 70, 64), "mixed"), ("diff_3D_lin_multixpu", (65, 66, 80), "mixed"),
])
def test_default_march(name, shape, resid):
    s, kw = S.SCRIPTS[name], {"itmax": 40, "nchk": 20, "resid": resid}
    a = run(s, shape, **kw)
    b = run(s, shape, {"warps2d": 2, "chunk2d": 32, "rows3d": 16, "chunk3d": 32}, **kw)
    assert a[1] >= a[2] and b[1] >= b[2]   # one launch per iteration
    assert np.array_equal(a[0], b[0])
