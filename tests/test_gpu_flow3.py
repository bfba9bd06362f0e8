"""The 3D FP64 kernel that holds whole steps: bit for bit the kernel of one
iteration per launch (which a context uses once a launch shape is set), where
tiles, rows, planes and warps are cut, at check cadences from every iteration
on, over several steps, and for fixed iteration counts."""
import numpy as np
import pytest

import ptdiff
from ptdiff import scripts as S

pytestmark = pytest.mark.gpu


def run(s, shape, march, iterate=0, steps=2, **kw):
    H0 = S.initial_condition(s, *shape)
    D = S.step_field(s, *shape) if s.model == S.LINSTEP else None
    with ptdiff.Solver(ptdiff.make_params(s, shape, **kw)) as sol:
        if march:
            sol.set_launch_config(rows3d=8, chunk3d=4)
        sol.set_state(H0, D)
        if iterate:
            sol.iterate(iterate)
            sol.iterate(iterate + 1)
            iters, eh = np.zeros(0), np.zeros(0)
        else:
            iters, eh = sol.step(steps)
        H = sol.get_state()
        sol.iterate(2)   # continues from the steps' H, Hold and fluxes
        return list(iters), eh, H, sol.get_state(), sol.counters()[0]


def compare(s, shape, **kw):
    a, b = run(s, shape, False, **kw), run(s, shape, True, **kw)
    assert a[0] == b[0]
    assert np.array_equal(a[2], b[2]) and np.array_equal(a[3], b[3])
    # the residual's cells are summed in another order: n 2^-53 relative at most
    assert len(a[1]) == len(b[1]) and np.allclose(a[1], b[1], rtol=np.prod(shape) * 2.0 ** -53, atol=0)
    return a, b


NAMES = ["diff_3D_lin_multixpu", "diff_3D_linstep_multixpu", "diff_3D_nonlin_multixpu"]


def fits(name, shape):
    """Whether the grid's tiles fit 151 SMs: 1 x 2 rows and planes with 28 warps
    each, LIN also 2 x 2 with 16."""
    nx, ny, nz = (n - 2 for n in shape)

    def warps(ry, rz):
        return -(-nx // 31) * -(-ny // ry) * -(-nz // rz)

    return warps(1, 2) <= 151 * 28 or ("_lin_" in name and warps(2, 2) <= 151 * 16)


# tiles of 1 x 1, 1 x 2 and 2 x 2 rows and planes, one tile to several in each direction
@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("shape", [(3, 130, 90), (4, 3, 2900), (33, 300, 4), (1100, 5, 7), (34, 32, 31), (70, 31, 18),
                                   (33, 60, 60), (40, 61, 62), (64, 40, 66), (64, 64, 64), (95, 52, 53), (35, 60, 70),
                                   (35, 95, 90)])
def test_flow3_step_is_the_march_step(name, shape):
    a, b = compare(S.SCRIPTS[name], shape, itmax=300)
    assert (a[4] < b[4]) == fits(name, shape)


@pytest.mark.parametrize("kw", [{"nchk": 1}, {"nchk": 3}, {"nchk": 7, "itmax": 47}, {"nchk": 64}, {"nchk": 50, "itmax": 30},
                                {"norm": "max"}, {"nchk": 4, "itmax": 4}])
@pytest.mark.parametrize("name,shape", [(NAMES[2], (36, 32, 29)), (NAMES[1], (40, 64, 64))])
def test_flow3_checks(name, shape, kw):
    compare(S.SCRIPTS[name], shape, **kw)


@pytest.mark.parametrize("k", [1, 2, 35])
@pytest.mark.parametrize("shape", [(40, 30, 28), (64, 62, 61)])
def test_flow3_iterate(shape, k):
    compare(S.SCRIPTS[NAMES[2]], shape, iterate=k)


def test_flow3_nan_is_reported():
    s = S.SCRIPTS[NAMES[2]]
    H0 = S.initial_condition(s, 40, 33, 30)
    H0[20, 15, 14] = np.nan
    with ptdiff.Solver(ptdiff.make_params(s, (40, 33, 30))) as sol:
        _, _, st = sol.solve(H0, raise_on_nan=False)
    assert st == ptdiff._abi.PTD_ENAN
