"""The march lengths chosen by grid size: a solve with the default launch shape
takes the same iterations and returns the same bits as one with a long march,
at sizes where the chosen march and the tiles leave remainders."""
import numpy as np
import pytest

import ptdiff
from ptdiff import scripts as S

pytestmark = pytest.mark.gpu

LONG = {"warps2d": 2, "chunk2d": 32, "rows3d": 16, "chunk3d": 32}


@pytest.mark.parametrize("name,shape,prec", [
    ("diff_2D_nonlin", (33, 34), "fp64"), ("diff_2D_linstep", (260, 251), "fp64"), ("diff_2D_lin", (95, 700), "fp64"),
    ("diff_2D_nonlin", (125, 131), "dfh"), ("diff_2D_lin", (64, 190), "df64"),
    ("diff_2D_nonlin", (121, 66), "fp32_rb"), ("diff_2D_linstep", (57, 259), "fp32_rb"),
    ("diff_3D_nonlin_multixpu", (33, 16, 5), "fp64"), ("diff_3D_linstep_multixpu", (32, 23, 66), "fp64"),
    ("diff_3D_nonlin_multixpu", (65, 31, 40), "dfh"), ("diff_3D_lin_multixpu", (34, 9, 67), "df64"),
    ("diff_3D_nonlin_multixpu", (63, 32, 35), "fp32_rb"),
])
def test_default_march_gives_the_long_march_solution(name, shape, prec):
    s = S.SCRIPTS[name]
    H0 = S.initial_condition(s, *shape)
    D = S.step_field(s, *shape) if s.model == S.LINSTEP else None
    got = []
    for cfg in (None, LONG):
        with ptdiff.Solver(ptdiff.make_params(s, shape, precision=prec, nt=2)) as sol:
            if cfg:
                sol.set_launch_config(**cfg)
            H = np.array(H0, order="F")
            iters, _, st = sol.solve(H, D)
            got.append((list(iters), H, st))
    assert got[0][2] == got[1][2] == 0
    assert got[0][0] == got[1][0]
    assert np.array_equal(got[0][1], got[1][1])
