"""Several 1D solvers alive at once, whose plans share one kernel and differ in
warps, window and shared memory: each returns the bits it returns alone."""
import threading

import numpy as np
import pytest

import ptdiff
from ptdiff import scripts as S

pytestmark = pytest.mark.gpu


def context(s, n):
    sol = ptdiff.Solver(ptdiff.make_params(s, (n,)))
    sol.set_state(S.initial_condition(s, n), S.step_field(s, n) if s.model == S.LINSTEP else None)
    return sol


def lone(s, n, steps):
    with context(s, n) as sol:
        its = [int(sol.step(1)[0][0]) for _ in range(steps)]
        return its, sol.get_state()


@pytest.mark.parametrize("name", ["diff_1D_lin", "diff_1D_linstep", "diff_1D_nonlin"])
@pytest.mark.parametrize("sizes", [(512, 64), (64, 1024), (1024, 512, 33), (9000, 7000)])
def test_contexts_step_in_turn(name, sizes):
    s = S.SCRIPTS[name]
    want = [lone(s, n, 2) for n in sizes]
    sols = [context(s, n) for n in sizes]   # all created before the first step
    its = [[] for _ in sizes]
    for _ in range(2):
        for k, sol in enumerate(sols):
            its[k].append(int(sol.step(1)[0][0]))
    for k, sol in enumerate(sols):
        assert its[k] == want[k][0] and np.array_equal(sol.get_state(), want[k][1])
        sol.close()


def test_contexts_are_created_while_others_step():
    s = S.SCRIPTS["diff_1D_lin"]
    sizes = [1024, 512, 200, 64]
    want = [lone(s, n, 2) for n in sizes]
    got = [[] for _ in sizes]

    def work(k):
        for _ in range(8):
            got[k].append(lone(s, sizes[k], 2))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(len(sizes)):
        assert len(got[k]) == 8
        assert all(its == want[k][0] and np.array_equal(H, want[k][1]) for its, H in got[k])
