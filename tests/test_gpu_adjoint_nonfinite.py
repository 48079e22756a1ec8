"""The advection adjoint's NaN and infinities: a node whose velocity or cotangent is not
finite spoils the gradient at all seven nodes of its stencil along each direction in which
it is weighted (the unused end too: its derivative is zero times that weight), and no
others."""
import numpy as np
import pytest

from tests.golden.cases import bubbles_case

pytestmark = pytest.mark.gpu
NI, NJ = 41, 37


def adjoint(gb, ua, va, lam):
    case = bubbles_case(NI, NJ, seed=4)
    c = gb.Context(NI, NJ)
    c.set(gb.FIELD_PHI, case["phi"])
    c.set(gb.FIELD_UA, ua)
    c.set(gb.FIELD_VA, va)
    mu = c.weno5_adjoint(0.3 / NI, lam)[0][2:-2, 2:-2]
    c.close()
    return mu


def cross(i, j, x, y):
    m = np.zeros((NJ, NI), bool)
    if x:
        m[j, i - 3:i + 4] = True
    if y:
        m[j - 3:j + 4, i] = True
    return m


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("where", ["ua", "va", "lam"])
@pytest.mark.parametrize("sign", [1, -1])
def test_nonfinite_weights_reach_the_whole_stencil(gb, where, value, sign):
    case = bubbles_case(NI, NJ, seed=4)
    rng = np.random.default_rng(7)
    ua, va = sign * (0.5 + np.abs(case["ua"])), sign * (0.5 + np.abs(case["va"]))
    lam = rng.uniform(0.5, 1.5, case["phi"].shape)
    i, j = 19, 17
    if where == "ua":  # the x-face between nodes i - 1 and i
        ua[j + 3, i + 3] = value
        want = cross(i - 1, j, True, False) | cross(i, j, True, False)
    elif where == "va":
        va[j + 3, i + 3] = value
        want = cross(i, j - 1, False, True) | cross(i, j, False, True)
    else:
        lam[j + 2, i + 2] = value
        want = cross(i, j, True, True)
    np.testing.assert_array_equal(~np.isfinite(adjoint(gb, ua, va, lam)), want)
