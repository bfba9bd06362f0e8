"""The one-launch 1D step: against the CPU oracle where windows, warps, CTAs
and the cluster are cut, at check cadences around its block length, and on the
first grid that no longer fits (one launch per iteration)."""
import numpy as np
import pytest

import ptdiff
from oracle import oracle as O
from ptdiff import scripts as S

pytestmark = pytest.mark.gpu

RTOL = 1e-10   # the parity bar of every FP64-accuracy form

LIMIT = 16 * 8 * (128 - 2 * 10)   # CTAs x warps x cells written back per window


def solve(s, n, **kw):
    H0 = S.initial_condition(s, n)
    D = S.step_field(s, n) if s.model == S.LINSTEP else None
    H = np.array(H0, order="F")
    with ptdiff.Solver(ptdiff.make_params(s, (n,), **kw)) as sol:
        iters, eh, _ = sol.solve(H, D)
    names = {"nchk": "nout"}
    okw = {names.get(k, k): v for k, v in kw.items()}
    if "norm" in okw:
        okw["norm"] = 1   # max
    Hr, itr, ehr, _ = O.solve(s, H0, D, **okw)
    return H, iters, eh, Hr, itr, ehr


@pytest.mark.parametrize("name", ["diff_1D_lin", "diff_1D_linstep", "diff_1D_nonlin"])
@pytest.mark.parametrize("n,kw", [(3, {}), (12, {}), (13, {}), (193, {}), (769, {}), (1409, {}),
                                  (64, {"nchk": 1}), (65, {"nchk": 7}), (300, {"nchk": 11}), (301, {"nchk": 64}),
                                  (90, {"norm": "max"})])
def test_line_step_matches_the_oracle(name, n, kw):
    kw = dict(nt=2, **kw)
    H, iters, eh, Hr, itr, ehr = solve(S.SCRIPTS[name], n, **kw)
    assert list(iters) == list(itr)
    assert np.linalg.norm(H - Hr) <= RTOL * np.linalg.norm(Hr)
    assert len(eh) == len(ehr)
    tol, at, nchk = S.SCRIPTS[name].tol, 0, kw.get("nchk", 10)
    for it in iters:   # a step's history: above tol until its last check
        n_chk = it // nchk
        assert np.all(eh[at : at + n_chk - 1] > tol)
        assert eh[at + n_chk - 1] <= tol
        at += n_chk


def one_launch_per_iteration(s, n, k):
    """H after k iterations by the kernel of one launch per iteration (which a
    solver with the consistent residual uses)."""
    with ptdiff.Solver(ptdiff.make_params(s, (n,), resid="consistent")) as sol:
        sol.set_state(S.initial_condition(s, n), S.step_field(s, n) if s.model == S.LINSTEP else None)
        sol.iterate(k)
        return sol.get_state()


@pytest.mark.parametrize("n,nchk,itmax", [(500, 10, 137), (LIMIT, 10, 60), (LIMIT + 1, 10, 60), (40, 50, 30)])
def test_line_step_stopped_by_itmax(n, nchk, itmax):
    """The checks leave no trace in the iterates: a step that reaches itmax
    returns the bits of that many iterations."""
    s = S.SCRIPTS["diff_1D_nonlin"]
    with ptdiff.Solver(ptdiff.make_params(s, (n,), nt=1, nchk=nchk, itmax=itmax)) as sol:
        sol.set_state(S.initial_condition(s, n))
        iters, eh = sol.step(1)
        H = sol.get_state()
    assert list(iters) == [itmax] and len(eh) == itmax // nchk
    assert np.array_equal(H, one_launch_per_iteration(s, n, itmax))


@pytest.mark.parametrize("name", ["diff_1D_lin", "diff_1D_linstep", "diff_1D_nonlin"])
@pytest.mark.parametrize("k", [1, 9, 10, 11, 37])
def test_line_iterate(name, k):
    s = S.SCRIPTS[name]
    with ptdiff.Solver(ptdiff.make_params(s, (333,))) as sol:
        sol.set_state(S.initial_condition(s, 333), S.step_field(s, 333) if s.model == S.LINSTEP else None)
        sol.iterate(k)
        sol.iterate(k)
        H = sol.get_state()
        assert sol.counters()[1] == 2 * k
    assert np.array_equal(H, one_launch_per_iteration(s, 333, 2 * k))
