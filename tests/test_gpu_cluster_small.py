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
