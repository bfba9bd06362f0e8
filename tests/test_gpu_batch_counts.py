"""Iteration counts of the defect-correction form on seeded nonlinear batches,
whose inner solves a last-bit change of the cell parameter e leads elsewhere:
the batch kernels fuse the root's argument over the product that they always
have (nonlin_cell_e).  The other product moves seven, eight and ten of the
counts below."""
import pytest

import ptdiff
from ptdiff import scripts as S

pytestmark = pytest.mark.gpu

COUNTS = {   # seed: iterations of the 24 instances
    10: [
        420, 110, 240, 120, 130, 110, 260, 430, 150, 580, 300, 120, 210, 220, 200, 370, 140, 230, 80, 330,
        110, 200, 110, 420],
    14: [
        430, 160, 210, 460, 260, 210, 240, 300, 140, 230, 360, 130, 250, 230, 150, 210, 120, 180, 350, 100,
        150, 410, 150, 180],
    18: [
        150, 330, 130, 110, 410, 160, 250, 160, 190, 120, 130, 310, 490, 260, 480, 60, 220, 290, 250, 160,
        110, 190, 270, 130],
}


@pytest.mark.parametrize("seed", sorted(COUNTS))
def test_defect_correction_counts(seed):
    sizes, Hs, _ = ptdiff.batch_instances(24, seed=seed, nmin=20, nmax=150)
    p = ptdiff.batch_params(24, model=S.NONLIN, precision="fp32_dc", nt=1, resc=1 / 1.2, itmax=2000)
    with ptdiff.BatchSolver(p, sizes, sizes) as b:
        iters, _ = b.solve(Hs)
    assert iters.ravel().tolist() == COUNTS[seed]
