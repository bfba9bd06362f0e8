"""The 3D rebased kernel of two cells per lane, at the edges of its 62 x 7
tiles, of the row pitch and of its march: bit for bit the two-iterations
kernel, which holds one cell per lane, and the FP64 solution of the step."""
import numpy as np
import pytest

import ptdiff
from ptdiff import scripts as S

pytestmark = pytest.mark.gpu


def solve(s, shape, **kw):
    H0 = S.initial_condition(s, *shape)
    H0 = np.asfortranarray(H0 + 0.05 * np.random.default_rng(3).random(shape))
    with ptdiff.Solver(ptdiff.make_params(s, shape, **kw)) as sol:
        sol.set_state(H0)
        iters, eh = sol.step(2)
        return list(iters), eh, sol.get_state()


@pytest.mark.parametrize("name", ["diff_3D_lin_multixpu", "diff_3D_nonlin_multixpu"])
@pytest.mark.parametrize("shape", [(3, 3, 3), (4, 9, 5), (32, 10, 18), (33, 8, 19), (62, 9, 20), (63, 16, 9), (64, 10, 8),
                                   (65, 9, 33), (66, 17, 7), (95, 12, 11), (96, 7, 40), (126, 23, 6), (127, 30, 20)])
def test_pair_kernel(name, shape):
    s = S.SCRIPTS[name]
    a = solve(s, shape, precision="fp32_rb", itmax=400)
    b = solve(s, shape, precision="fp32_rb", itmax=400, rb_tblock_3d=True)
    assert a[0] == b[0] and np.array_equal(a[2], b[2])


@pytest.mark.parametrize("name,shape,march", [("diff_3D_lin_multixpu", (70, 40, 50), m) for m in (1, 5, 48, 300)]
                         + [("diff_3D_nonlin_multixpu", (64, 30, 41), m) for m in (1, 7, 39, 100)])
def test_pair_kernel_marches(name, shape, march):
    """A march of any length gives the same bits."""
    s = S.SCRIPTS[name]
    H0 = S.initial_condition(s, *shape)
    out = []
    for m in (None, march):
        with ptdiff.Solver(ptdiff.make_params(s, shape, precision="fp32_rb")) as sol:
            if m:
                sol.set_launch_config(chunk3d=m)
            sol.set_state(H0)
            sol.iterate(21)
            out.append(sol.get_state())
    assert np.array_equal(out[0], out[1])


# the first grids above the line where the one-cell kernel takes 16-row CTAs
def test_large_one_cell_kernel_is_the_two_iterations_kernel():
    s = S.SCRIPTS["diff_3D_nonlin_multixpu"]
    shape = (137, 134, 132)
    a = solve(s, shape, precision="fp32_rb", itmax=40)
    b = solve(s, shape, precision="fp32_rb", itmax=40, rb_tblock_3d=True)
    assert a[0] == b[0] and np.array_equal(a[2], b[2])


@pytest.mark.parametrize("shape", [(137, 134, 132), (133, 136, 132)])
def test_one_cell_kernel_above_and_below_the_line(shape):
    """Either solver stops a step at an RMS residual of tol, so the solutions
    differ by dt 2 tol at most (the step's operator is at least 1/dt)."""
    s = S.SCRIPTS["diff_3D_linstep_multixpu"]
    out = []
    for prec in ("fp64", "fp32_rb"):
        H = S.initial_condition(s, *shape)
        with ptdiff.Solver(ptdiff.make_params(s, shape, precision=prec, nt=1)) as sol:
            sol.solve(H, S.step_field(s, *shape))
        out.append(H)
    assert np.sqrt(np.mean((out[0] - out[1]) ** 2)) <= s.dt * 2 * s.tol
