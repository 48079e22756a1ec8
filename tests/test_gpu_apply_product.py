"""The operator product's integer-pipe form, which grids of 2^21 cells and more take under the
FP32 preconditioner: a solve to 1e-8 at 2048 x 1024 (the first size that takes it) and one
column narrower (which does not), each in one pass (the true residual agrees with the CG's) and
against the FP64 solve, whose product takes the plain form."""
import numpy as np
import pytest

from test_gpu_cluster_tail import case_for, make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ni,nj", [(2048, 1024), (2047, 1024)])
def test_solve_meets_its_residual(gb, ni, nj):
    case = case_for(ni, nj, 3)
    c = make(gb, case, True)
    bx, by, dg, rhs = c.poisson_assemble(0.5 / (ni - 1))
    x, st = c.poisson_solve(rhs, opts=gb.solve_opts(precision=gb.PRECISION_MIXED, tolerance=1e-8))
    y, sty = c.poisson_solve(rhs, opts=gb.solve_opts(precision=gb.PRECISION_FP64, tolerance=1e-8))
    c.close()
    assert st.rel_residual <= 1e-8 and st.outer_iterations == 1
    # both precisions' iterates meet the same residual; p differs by the solve tolerance's share
    assert np.linalg.norm(x - y) <= 1e-5 * np.linalg.norm(y)
    assert abs(st.iterations - sty.iterations) <= max(2, 0.15 * sty.iterations)
