"""The FP64 rebase of the rebased FP32 form where its march and its integer
arithmetic can go wrong: grids at the march's and tile's remainders, fields
with exact zeros, negative values and wide exponents (which take the FP64
arithmetic beside the integer one), against the FP64 solver.

A step stops when the FP64 residual of the state is at tol in RMS, for either
solver, so the two solutions differ by at most the change that a residual of
2 tol makes in an implicit step: dt 2 tol in RMS (the step's operator is at
least 1/dt)."""
import numpy as np
import pytest

import ptdiff
from ptdiff import scripts as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,shape", [
    ("diff_2D_lin", (33, 34)), ("diff_2D_linstep", (64, 257)), ("diff_2D_nonlin", (70, 129)), ("diff_2D_lin", (97, 31)),
    ("diff_3D_lin_multixpu", (33, 9, 18)), ("diff_3D_linstep_multixpu", (40, 17, 33)),
    ("diff_3D_nonlin_multixpu", (31, 16, 35)),
])
def test_rebased_solution_on_rough_fields(name, shape):
    s = S.SCRIPTS[name]
    rng = np.random.default_rng(2)
    H0 = S.initial_condition(s, *shape)
    if s.model != S.NONLIN:
        H0 = H0 - 0.3                                            # both signs
        H0[rng.random(shape) < 0.1] = 0.0
        H0[rng.random(shape) < 0.1] *= 1e-70
    H0 = np.asfortranarray(H0)
    D = S.step_field(s, *shape) if s.model == S.LINSTEP else None
    out = []
    for prec in ("fp64", "fp32_rb"):
        H = np.array(H0, order="F")
        with ptdiff.Solver(ptdiff.make_params(s, shape, precision=prec, nt=1)) as sol:
            sol.solve(H, D)
        out.append(H)
    rms = np.sqrt(np.mean((out[0] - out[1]) ** 2))
    assert rms <= s.dt * 2 * s.tol
