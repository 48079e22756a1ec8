"""The cluster tail's windows (a CTA's row stripe plus the halo that one side of smoothing
uses up) against the single-CTA tail: one V-cycle on grids whose rows split unevenly over
the CTAs, whose rows are odd, whose halos reach past the neighbouring stripe or the walls,
and that hold one, two or three distributed levels, for one to three sweeps a side.  The
two tails differ by the rounding of the dense coarse solve and of the levels that the
smaller single-CTA tail leaves to the tiled launches (tolerances as
tests/test_gpu_cluster_tail.py's first step)."""
import numpy as np
import pytest

from test_gpu_cluster_tail import case_for, make, rel_l2, system

pytestmark = pytest.mark.gpu
SHAPES = [(64, 64), (65, 67), (130, 126), (63, 260), (128, 128), (40, 400), (33, 95)]


@pytest.mark.parametrize("ni,nj", SHAPES)
@pytest.mark.parametrize("prec_name", ["FP64", "MIXED"])
def test_vcycle_matches_single_cta_tail(gb, ni, nj, prec_name):
    prec = getattr(gb, "PRECISION_" + prec_name)
    case = case_for(ni, nj, 7)
    r = np.random.default_rng(ni + nj).standard_normal((nj, ni))
    tol = 1e-11 if prec_name == "FP64" else 2e-5
    z = {}
    for cluster in (True, False):
        c = make(gb, case, cluster)
        system(gb, c, 0.5 / (max(ni, nj) - 1))
        z[cluster] = [c.preconditioner_apply(r, prec, nu) for nu in (1, 2, 3)]
        c.close()
    for a, b in zip(z[True], z[False]):
        assert np.all(np.isfinite(a)) and np.linalg.norm(a) > 0
        assert rel_l2(a, b) <= tol
