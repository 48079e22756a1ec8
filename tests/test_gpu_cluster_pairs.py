"""The cluster tail where a thread owns three cell pairs (FP64: its largest kernel), with one
to three sweeps a side: one V-cycle against the single-CTA tail, to the tolerance of
tests/test_gpu_cluster_windows.py from the 128^2 levels down and to the last bit from the
64^2 ones, and a whole solve.  Wide FP64 levels of few rows, which would take more than two
pairs with two sweeps in the 64^2 form, stay with the single-CTA tail."""
import numpy as np
import pytest

from test_gpu_cluster_tail import case_for, make, rel_l2, system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ni,nj,small", [(111, 80, False), (121, 132, False), (72, 116, False), (126, 69, False),
                                         (142, 15, True), (615, 64, True), (346, 39, True)])
def test_three_pairs_match_the_single_cta_tail(gb, ni, nj, small):
    case = case_for(ni, nj, 9)
    got = {}
    for cluster in (True, False):
        c = make(gb, case, cluster)
        rhs = system(gb, c, 0.5 / (max(ni, nj) - 1))
        assert (c.solver_layout(gb.PRECISION_FP64)[1] >= 0) == cluster
        r = rhs + np.random.default_rng(ni * nj).standard_normal((nj, ni)) * np.abs(rhs).max() * 1e-3
        got[cluster] = [c.preconditioner_apply(r, gb.PRECISION_FP64, nu) for nu in (1, 2, 3)]
        x, st = c.poisson_solve(rhs, opts=gb.solve_opts(precision=gb.PRECISION_FP64, tolerance=1e-9, mg_smooth=3))
        assert st.rel_residual <= 1e-9
        if small:
            got[cluster].append(x)
        c.close()
    for a, b in zip(got[True], got[False]):
        assert np.all(np.isfinite(a)) and np.linalg.norm(a) > 0
        assert np.array_equal(a, b) if small else rel_l2(a, b) <= 1e-11


@pytest.mark.parametrize("ni,nj", [(1000, 16), (902, 18), (595, 22)])
def test_wide_fp64_levels_of_few_rows_stay_in_one_cta(gb, ni, nj):
    c = make(gb, case_for(ni, nj, 3), True)
    assert c.solver_layout(gb.PRECISION_FP64)[1] == -1
    assert c.solver_layout(gb.PRECISION_MIXED)[1] >= 0
    c.close()
