"""The marches taken with checks (nearly) every iteration: the same iterations
and bits as with another march, on both sides of the cadence where they begin
and where tiles and marches leave remainders."""
import numpy as np
import pytest

import ptdiff
from ptdiff import scripts as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nchk", [1, 3, 4])
@pytest.mark.parametrize("name,shape,prec", [
    ("diff_3D_lin_multixpu", (33, 16, 23), "fp32_dc"), ("diff_3D_linstep_multixpu", (95, 50, 67), "fp32_dc"),
    ("diff_3D_nonlin_multixpu", (130, 62, 35), "fp32_dc"), ("diff_2D_linstep", (97, 131), "dfh"),
    ("diff_2D_linstep", (1000, 1001), "df64"),
])
def test_march_of_frequent_checks(name, shape, prec, nchk):
    s = S.SCRIPTS[name]
    H0 = S.initial_condition(s, *shape)
    D = S.step_field(s, *shape) if s.model == S.LINSTEP else None
    out = []
    for cfg in (None, {"warps2d": 4, "chunk2d": 16, "chunk3d": 5}):
        with ptdiff.Solver(ptdiff.make_params(s, shape, precision=prec, nchk=nchk, itmax=48, tol=1e-300)) as sol:
            if cfg:
                sol.set_launch_config(**cfg)
            sol.set_state(H0, D)
            iters, _ = sol.step(1)
            out.append((list(iters), sol.get_state()))
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1])
