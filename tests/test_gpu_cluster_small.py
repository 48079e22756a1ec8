"""The cluster tail from the 64^2 levels down, which FP64 hierarchies take whose 128^2 level
does not fit a CTA: the launches that it replaces (tiled levels, the single-CTA tail) add
and round in the same order, so one V-cycle gives the same bits, for one to three sweeps a
side, on grids whose small levels have even and odd rows and columns.  128 x 500 keeps the
tail from its larger level down, whose dense solve is summed in another order (tolerance as
tests/test_gpu_cluster_windows.py)."""
import numpy as np
import pytest

from test_gpu_cluster_tail import case_for, make, rel_l2, system

pytestmark = pytest.mark.gpu
SHAPES = [(130, 126), (253, 190), (257, 250), (511, 385), (500, 376), (128, 500)]


@pytest.mark.parametrize("ni,nj", SHAPES)
def test_vcycle_has_the_single_cta_tails_bits(gb, ni, nj):
    case = case_for(ni, nj, 5)
    r = np.random.default_rng(ni * nj).standard_normal((nj, ni))
    z = {}
    for cluster in (True, False):
        c = make(gb, case, cluster)
        system(gb, c, 0.5 / (max(ni, nj) - 1))
        z[cluster] = [c.preconditioner_apply(r, gb.PRECISION_FP64, nu) for nu in (1, 2, 3)]
        if cluster:
            top = c.solver_layout(gb.PRECISION_FP64)[1]
        c.close()
    small = top >= 0 and -(-ni // 2**top) * -(-nj // 2**top) <= 64 * 64
    assert small == ((ni, nj) != (128, 500))
    for a, b in zip(z[True], z[False]):
        assert np.all(np.isfinite(a)) and np.linalg.norm(a) > 0
        assert np.array_equal(a, b) if small else rel_l2(a, b) <= 1e-11


# Grids that the 64^2 form holds whole (r.z summed by its first CTA), over the numbers of CTAs
# that their rows allow (16, 8, 4, 1), one of more levels with its tail at 40 x 30, and the
# smallest ones: whole solves, both precisions.  8 x 120 is the larger form's (64 rows and
# up): its V-cycles to the tolerances of tests/test_gpu_cluster_windows.py.
@pytest.mark.parametrize("ni,nj", [(64, 48), (65, 63), (40, 32), (41, 31), (63, 17), (100, 15), (16, 9), (24, 8), (9, 9), (8, 120), (640, 480)])
@pytest.mark.parametrize("prec_name", ["FP64", "MIXED"])
def test_solve_has_the_single_cta_tails_bits(gb, ni, nj, prec_name):
    prec = getattr(gb, "PRECISION_" + prec_name)
    case = case_for(ni, nj, 3)
    got = {}
    for cluster in (True, False):
        c = make(gb, case, cluster)
        rhs = system(gb, c, 0.5 / (max(ni, nj) - 1))
        r = rhs + np.random.default_rng(ni * nj).standard_normal((nj, ni)) * np.abs(rhs).max() * 1e-3
        got[cluster] = [c.preconditioner_apply(r, prec, nu) for nu in (1, 2, 3)]
        for nu in (1, 2, 3):
            x, st = c.poisson_solve(rhs, opts=gb.solve_opts(precision=prec, tolerance=1e-9, mg_smooth=nu), allow_max_iters=True)
            got[cluster] += [x, np.array([st.iterations, st.outer_iterations])]
        c.close()
    if (ni, nj) == (8, 120):
        for a, b in zip(got[True][:3], got[False][:3]):
            assert np.all(np.isfinite(a)) and rel_l2(a, b) <= (1e-11 if prec_name == "FP64" else 2e-5)
        return
    for a, b in zip(got[True], got[False]):
        assert np.all(np.isfinite(a)) and np.array_equal(a, b)
