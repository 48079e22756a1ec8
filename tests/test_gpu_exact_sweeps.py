"""The exact FP64 level-set sweeps against the CPU oracle, bit for bit, where their tiles
and their choice of arithmetic can go wrong: grids at and beside the 32 x 4 tiles' edges,
level sets with kinks, plateaus and exact zeros (nodes that need both one-sided
derivatives), and magnitudes or a WENO epsilon outside the range of the fast arithmetic."""
import numpy as np
import pytest

from tests.golden.cases import bubbles_case

pytestmark = pytest.mark.gpu
SIZES = [(4, 4), (5, 9), (31, 3 + 1), (32, 4), (33, 5), (64, 8), (65, 13), (97, 7)]


def level_set(kind, ni, nj):
    c = bubbles_case(ni, nj, seed=ni + nj)
    phi = c["phi"]
    X, Y = np.meshgrid(np.linspace(-1, 1, ni + 4), np.linspace(-1, 1, nj + 4))
    if kind == "kink":
        phi = np.minimum(np.abs(X) - 0.3, 0.4 - np.abs(Y))
    elif kind == "plateau":
        phi = np.clip(phi, -0.02, 0.05)
        phi[np.abs(phi) < 0.01] = 0.0
    elif kind == "noise":
        phi = np.random.default_rng(ni).uniform(-1, 1, phi.shape)
    elif kind == "large":
        phi = phi * 1e40
    elif kind == "small":
        phi = phi * 1e-120
    return np.ascontiguousarray(phi), c


@pytest.mark.parametrize("kind,eps", [("circles", 1e-6), ("kink", 1e-6), ("plateau", 1e-6), ("noise", 1e-6), ("large", 1e-6),
                                      ("small", 1e-6), ("circles", 1e-40)])
@pytest.mark.parametrize("ni,nj", SIZES)
def test_exact_sweeps_equal_the_oracle(gb, oracle, ni, nj, kind, eps):
    phi, case = level_set(kind, ni, nj)
    g, pr = oracle.grid(ni, nj), oracle.params(weno_epsilon=eps, reinit_iterations=3)
    dt = 0.3 / max(ni, nj)
    c = gb.Context(ni, nj, weno_epsilon=eps, reinit_iterations=3)
    c.set(gb.FIELD_PHI, phi)
    c.set(gb.FIELD_UA, case["ua"])
    c.set(gb.FIELD_VA, case["va"])
    want = phi.copy()
    c.levelset_advection(dt)
    oracle.levelset_advection(g, pr, want, case["ua"].copy(), case["va"].copy(), dt)
    np.testing.assert_array_equal(c.get(gb.FIELD_PHI), want)
    c.set(gb.FIELD_PHI, phi)
    want = phi.copy()
    c.reinitialization()
    oracle.reinitialization(g, pr, want)
    np.testing.assert_array_equal(c.get(gb.FIELD_PHI), want)
    c.close()


def test_integer_pipe_arithmetic_rounds_as_ieee(gb):
    assert gb.check_exact_division(1 << 22, seed=9) == 0
