"""The one-launch 2D step: bit for bit the kernel of one iteration per launch
(which a context uses once a launch shape is set), where tiles, rows and warps
are cut, at check cadences from every iteration on, and from several threads."""
import threading

import numpy as np
import pytest

import ptdiff
from ptdiff import scripts as S

pytestmark = pytest.mark.gpu


def fields(s, shape):
    return S.initial_condition(s, *shape), S.step_field(s, *shape) if s.model == S.LINSTEP else None


def run(s, shape, march, iterate=0, **kw):
    H0, D = fields(s, shape)
    with ptdiff.Solver(ptdiff.make_params(s, shape, **kw)) as sol:
        if march:
            sol.set_launch_config(warps2d=2, chunk2d=8)
        sol.set_state(H0, D)
        if iterate:
            sol.iterate(iterate)
            sol.iterate(iterate + 1)
            iters, eh = np.zeros(0), np.zeros(0)
        else:
            iters, eh = sol.step(2)
        return list(iters), eh, sol.get_state(), sol.counters()[0]


def compare(s, shape, **kw):
    a, b = run(s, shape, False, **kw), run(s, shape, True, **kw)
    assert a[0] == b[0]
    assert np.array_equal(a[2], b[2])
    # the residual's cells are summed in another order: n 2^-53 relative at most
    assert len(a[1]) == len(b[1]) and np.allclose(a[1], b[1], rtol=shape[0] * shape[1] * 2.0 ** -53, atol=0)
    return a, b


@pytest.mark.parametrize("name", ["diff_2D_lin", "diff_2D_linstep", "diff_2D_nonlin"])
@pytest.mark.parametrize("shape", [(3, 3), (4, 3), (3, 40), (33, 33), (34, 31), (64, 65), (65, 64), (95, 190)])
def test_flow_step_is_the_march_step(name, shape):
    a, b = compare(S.SCRIPTS[name], shape)
    assert a[3] < b[3]   # one launch per step


# rows per tile 1, 2, 3, 4, 6 and the first grid that does not fit (152 SMs)
# (of these grids: 1, 2, 3, 4, 5 rows and one that does not fit; 6 rows: test_gpu_plans.py)
@pytest.mark.parametrize("name,shape", [("diff_2D_nonlin", (300, 280)), ("diff_2D_linstep", (500, 333)),
                                        ("diff_2D_lin", (512, 512)), ("diff_2D_nonlin", (600, 521)),
                                        ("diff_2D_linstep", (701, 643)), ("diff_2D_nonlin", (900, 800))])
def test_flow_tile_heights(name, shape):
    compare(S.SCRIPTS[name], shape, itmax=60, nchk=20)


@pytest.mark.parametrize("kw", [{"nchk": 1}, {"nchk": 3}, {"nchk": 7, "itmax": 47}, {"nchk": 64}, {"nchk": 50, "itmax": 30},
                                {"norm": "max"}, {"nchk": 4, "itmax": 4}])
@pytest.mark.parametrize("name,shape", [("diff_2D_nonlin", (70, 41)), ("diff_2D_linstep", (40, 97))])
def test_flow_checks(name, shape, kw):
    compare(S.SCRIPTS[name], shape, **kw)


@pytest.mark.parametrize("k", [1, 2, 35])
def test_flow_iterate(k):
    compare(S.SCRIPTS["diff_2D_nonlin"], (100, 67), iterate=k)


def test_flow_nan_is_reported():
    s = S.SCRIPTS["diff_2D_nonlin"]
    H0, _ = fields(s, (80, 70))
    H0[40, 30] = np.nan
    with ptdiff.Solver(ptdiff.make_params(s, (80, 70))) as sol:
        _, _, st = sol.solve(H0, raise_on_nan=False)
    assert st == ptdiff._abi.PTD_ENAN


def test_flow_from_several_threads():
    """Contexts stepping at the same time on one GPU: each launch needs all its
    CTAs resident, and none may wait for another's for good."""
    s = S.SCRIPTS["diff_2D_nonlin"]
    shapes = [(128, 128), (200, 150), (90, 260)]
    want = [run(s, sh, False)[2] for sh in shapes]
    got = [[] for _ in shapes]

    def work(k):
        for _ in range(5):
            got[k].append(run(s, shapes[k], False)[2])

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(shapes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(len(shapes)):
        assert len(got[k]) == 5 and all(np.array_equal(g, want[k]) for g in got[k])
