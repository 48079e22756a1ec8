"""The curvature of a level set with infinities, NaN and magnitudes whose squares overflow or
vanish, against the CPU oracle, bit for bit: where the curvature is NaN the reference's clamp
stores nothing (LEVELSET_2D.h:980-988) and the field keeps its value, here the initial zero."""
import numpy as np
import pytest

from tests.golden.cases import bubbles_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 1e300, -1e155, 1e-300, 5e-324])
@pytest.mark.parametrize("ni,nj", [(33, 20), (64, 41)])
def test_curvature_equals_the_oracle(gb, oracle, ni, nj, value):
    phi = bubbles_case(ni, nj, seed=6)["phi"]
    rng = np.random.default_rng(ni)
    phi[rng.random(phi.shape) < 0.02] = value
    c = gb.Context(ni, nj)
    c.set(gb.FIELD_PHI, phi)
    c.curvature()
    got = c.get(gb.FIELD_KAPPA)
    c.close()
    want = np.zeros((nj, ni))
    oracle.curvature(oracle.grid(ni, nj), phi.copy(), want)
    np.testing.assert_array_equal(got, want)
    assert np.all(np.isfinite(got))
