"""The tiled level-set and velocity kernels on grids of more tile rows than one launch holds
(65535): the last 600 rows of a tall grid equal a 600-row grid that holds the same rows, bit
for bit (every update is local; cell sizes are powers of two), both precisions; rows near the
cut are left out."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
H = 2.0**-10  # cell size


def fields(gb, ni, nj):
    rng = np.random.default_rng(nj)
    c = gb.Context(ni, nj, 0.0, 0.0, (ni - 1) * H, (nj - 1) * H)
    f = {k: rng.uniform(-1, 1, c.shape(getattr(gb, "FIELD_" + k))) for k in ("U", "V", "UA", "VA")}
    c.close()
    i, j = np.meshgrid(np.arange(ni + 4), np.arange(nj + 4))
    f["PHI"] = 0.01 * np.sin(0.05 * j) + 3e-3 * np.cos(0.7 * i + 0.01 * j) + 1e-5 * rng.uniform(-1, 1, (nj + 4, ni + 4))
    return f


def run(gb, f, ni, nj, prec, what):
    c = gb.Context(ni, nj, 0.0, 0.0, (ni - 1) * H, (nj - 1) * H, reinit_iterations=2, advection_precision=prec)
    c.set_flow_params(water_viscosity=1.0, air_viscosity=0.01, viscosity=True)
    for k, a in f.items():
        c.set(getattr(gb, "FIELD_" + k), np.ascontiguousarray(a))
    if what in ("levelset", "advection"):
        c.levelset_advection(0.2 * H)
        if what == "levelset":
            c.reinitialization()
        out = [c.get(gb.FIELD_PHI)]
    else:
        c.velocity_advection(0.1 * H)
        c.sourcing(1e-8)
        out = [c.get(gb.FIELD_U), c.get(gb.FIELD_V)]
    c.close()
    return out


# 262140 rows are 65535 tiles of 4, 524280 of 8 (the mixed reinitialisation's limit).
@pytest.mark.parametrize("what,prec,nj", [("levelset", 0, 262140), ("levelset", 0, 262141), ("levelset", 0, 300001), ("advection", 1, 524281), ("levelset", 1, 262141),
                                          ("velocity", 0, 524281), ("velocity", 1, 524400)])
def test_rows_beyond_one_launch(gb, what, prec, nj):
    ni, short = 5, 600
    f = fields(gb, ni, nj)
    tall = run(gb, f, ni, nj, prec, what)
    ref = run(gb, {k: a[nj - short:] for k, a in f.items()}, ni, short, prec, what)
    for a, b in zip(tall, ref):
        np.testing.assert_array_equal(a[nj - short:][40:], b[40:])
        assert not np.array_equal(a[nj - short:][40:-40], f["U" if what == "velocity" else "PHI"][nj - short:][40:-40])
