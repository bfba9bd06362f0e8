"""Several physical steps per call, which the 1D and 2D FP64 kernels take in one
launch: bit for bit the steps taken one per call, with the same iteration
counts, residual histories and counters."""
import numpy as np
import pytest

import ptdiff
from ptdiff import scripts as S

pytestmark = pytest.mark.gpu


def run(s, shape, calls, Hold=False, **kw):
    H0 = S.initial_condition(s, *shape)
    D = S.step_field(s, *shape) if s.model == S.LINSTEP else None
    with ptdiff.Solver(ptdiff.make_params(s, shape, **kw)) as sol:
        if Hold:
            sol.solve(np.array(H0, order="F"), D, Hold=np.asfortranarray(0.5 * H0 + 0.25))
        else:
            sol.set_state(H0, D)
        out = [sol.step(n) for n in calls]
        launches, iterations = sol.counters()
        H = sol.get_state()
        sol.iterate(3)   # continues from the steps' H, Hold and fluxes
        return (np.concatenate([o[0] for o in out]), np.concatenate([o[1] for o in out]), H, sol.get_state(),
                iterations, launches)


def compare(s, shape, n, **kw):
    a, b = run(s, shape, [n], **kw), run(s, shape, [1] * n, **kw)
    for x, y in zip(a[:4], b[:4]):
        assert np.array_equal(x, y)
    assert a[4] == b[4]
    return a, b


@pytest.mark.parametrize("name,shape", [("diff_1D_lin", (64,)), ("diff_1D_linstep", (769,)), ("diff_1D_nonlin", (5000,)),
                                        ("diff_2D_lin", (3, 3)), ("diff_2D_linstep", (34, 31)),
                                        ("diff_2D_nonlin", (65, 64)), ("diff_2D_linstep", (300, 280)),
                                        ("diff_2D_nonlin", (400, 421)), ("diff_2D_lin", (512, 512)),
                                        ("diff_2D_nonlin", (600, 521)), ("diff_2D_nonlin", (700, 600)),
                                        ("diff_2D_linstep", (701, 603)), ("diff_2D_lin", (760, 680))])
@pytest.mark.parametrize("kw", [{}, {"nchk": 7}])
def test_steps_of_one_launch(name, shape, kw):
    a, b = compare(S.SCRIPTS[name], shape, 4, **kw)
    assert a[5] == b[5] - 3


@pytest.mark.parametrize("name,shape", [("diff_1D_nonlin", (90,)), ("diff_2D_nonlin", (70, 41))])
@pytest.mark.parametrize("kw", [{"nchk": 1}, {"nchk": 1, "norm": "max"}, {"Hold": True}, {"nchk": 3, "itmax": 25},
                                {"nchk": 10, "itmax": 8}, {"nchk": 5000, "itmax": 5000}])
def test_steps_at_the_limits_of_a_launch(name, shape, kw):
    """History past the host's part, a separate first Hold, steps stopped by
    itmax (with and without iterations after the last check), long cadences."""
    compare(S.SCRIPTS[name], shape, 5, **kw)


@pytest.mark.parametrize("name,shape", [("diff_1D_lin", (20,)), ("diff_2D_lin", (12, 9))])
def test_more_steps_than_a_launch_takes(name, shape):
    a, b = compare(S.SCRIPTS[name], shape, 300)
    assert a[5] < b[5] - 250


@pytest.mark.parametrize("name,shape", [("diff_1D_nonlin", (80,)), ("diff_2D_nonlin", (80, 70))])
def test_nan_ends_the_steps(name, shape):
    s = S.SCRIPTS[name]
    H0 = S.initial_condition(s, *shape)
    H0[tuple(n // 2 for n in shape)] = np.nan
    with ptdiff.Solver(ptdiff.make_params(s, shape, nt=6)) as sol:
        iters, _, st = sol.solve(H0, raise_on_nan=False)
    assert st == ptdiff._abi.PTD_ENAN and iters[0] > 0 and not iters[1:].any()


@pytest.mark.parametrize("name,shape", [("diff_1D_nonlin", (70,)), ("diff_2D_nonlin", (64, 41)), ("diff_2D_nonlin", (61, 40)),
                                        ("diff_3D_nonlin_multixpu", (32, 9, 10)), ("diff_3D_nonlin_multixpu", (35, 9, 10))])
@pytest.mark.parametrize("kw", [{}, {"precision": "df64"}, {"precision": "dfh"}, {"precision": "fp32_rb"}, {"autotune": True}])
def test_a_new_state_leaves_nothing_of_the_last(name, shape, kw):
    """With rows that fill the pitch and rows that do not, after steps from
    another state and after the autotuner's: bit for bit a fresh context."""
    s = S.SCRIPTS[name]
    H0 = S.initial_condition(s, *shape)
    out = []
    for used in (False, True):
        with ptdiff.Solver(ptdiff.make_params(s, shape, **dict(kw, autotune=kw.get("autotune", False) and used))) as sol:
            if used:
                sol.set_state(np.asfortranarray(2.0 * H0 + 1.0))
                sol.step(1)
                sol.iterate(3)
            sol.set_state(H0)
            sol.iterate(15)
            out.append(sol.get_state())
    assert np.array_equal(out[0], out[1])
