"""The tiled ENO3 advection and viscous stage against the CPU oracle at and beside the
edges of their 32 x 8 tiles, with magnitudes inside and outside the range of the exact
products on the integer pipes, zeros, and a density and viscosity band (and none).  The
advection is bit-exact; the viscous faces are held to 1e-13 relative, the difference that
the smeared Heaviside's sine makes (exact where no node lies in the band)."""
import numpy as np
import pytest

from tests.golden.cases import bubbles_case

pytestmark = pytest.mark.gpu
SIZES = [(4, 4), (7, 31), (31, 8), (32, 7), (33, 16), (63, 9), (64, 24)]
FIELDS = ("u", "v", "ua", "va")


def case_of(ni, nj, scale):
    c = bubbles_case(ni, nj, seed=3 * ni + nj)
    for k in ("u", "v", "ua", "va"):
        c[k] = c[k] * scale
        c[k][:, : c[k].shape[1] // 3] = 0.0
    return c


def context(gb, c, ni, nj):
    x = gb.Context(ni, nj)
    for f, k in ((gb.FIELD_PHI, "phi"), (gb.FIELD_U, "u"), (gb.FIELD_V, "v"), (gb.FIELD_UA, "ua"), (gb.FIELD_VA, "va")):
        x.set(f, c[k])
    return x


@pytest.mark.parametrize("scale", [1.0, 1e-70, 1e-150, 1e70])
@pytest.mark.parametrize("ni,nj", SIZES)
def test_velocity_advection_equals_the_oracle(gb, oracle, ni, nj, scale):
    c = case_of(ni, nj, scale)
    dt = 0.3 / (max(ni, nj) * max(scale, 1.0))
    x = context(gb, c, ni, nj)
    x.velocity_advection(dt)
    w = {k: c[k].copy() for k in FIELDS}
    oracle.velocity_advection(oracle.grid(ni, nj), oracle.params(), w["u"], w["v"], w["ua"], w["va"], dt)
    for f, k in ((gb.FIELD_U, "u"), (gb.FIELD_V, "v"), (gb.FIELD_UA, "ua"), (gb.FIELD_VA, "va")):
        np.testing.assert_array_equal(x.get(f), w[k], err_msg=k)
    x.close()


@pytest.mark.parametrize("scale", [1.0, 1e-70])
@pytest.mark.parametrize("band", [True, False])
@pytest.mark.parametrize("ni,nj", SIZES)
def test_viscosity_equals_the_oracle(gb, oracle, ni, nj, band, scale):
    c = case_of(ni, nj, scale)
    if not band:
        c["phi"][:] = 10.0
    visc = dict(water_viscosity=1.0, air_viscosity=0.0)
    dt = 0.01 / max(ni, nj) ** 2
    x = context(gb, c, ni, nj)
    x.set_flow_params(viscosity=True, **visc)
    x.sourcing(dt)
    u, v = c["u"].copy(), c["v"].copy()
    oracle.sourcing(oracle.grid(ni, nj), oracle.params(), oracle.flow(viscosity=True, **visc), c["phi"].copy(), u, v, None, dt)
    for f, want in ((gb.FIELD_U, u), (gb.FIELD_V, v)):
        got = x.get(f)
        if band:
            np.testing.assert_allclose(got, want, rtol=1e-13, atol=1e-13 * np.abs(want).max())
        else:
            np.testing.assert_array_equal(got, want)
    x.close()
