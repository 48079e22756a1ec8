"""One exact FP64 reinitialisation sweep for every S that a caller may hand to
gb2d_reinit_sweep_apply, bit for bit against the same operations in numpy: S of ordinary
size, at and beside the ends of the fast arithmetic's range (2^-100, 2^100), so large that
the update overflows, infinite, NaN and zero."""
import numpy as np
import pytest

from tests.golden.cases import bubbles_case

pytestmark = pytest.mark.gpu


def weno(a1, a2, a3, a4, a5, eps):
    c13, q = 13.0 / 12.0, 0.25
    A1, B1 = a1 - 2 * a2 + a3, a1 - 4 * a2 + 3 * a3
    A2, B2 = a2 - 2 * a3 + a4, a2 - a4
    A3, B3 = a3 - 2 * a4 + a5, 3 * a3 - 4 * a4 + a5
    e1, e2, e3 = (eps + (c13 * A * A + q * B * B) for A, B in ((A1, B1), (A2, B2), (A3, B3)))
    l1, l2, l3 = (1.0 / 10.0) / (e1 * e1), (6.0 / 10.0) / (e2 * e2), (3.0 / 10.0) / (e3 * e3)
    s = l1 + l2 + l3
    return (l1 / s * (a1 / 3 - a2 * 7 / 6 + a3 * 11 / 6) + l2 / s * (a2 * ((-1.0) / 6.0) + a3 * 5 / 6 + a4 / 3) +
            l3 / s * (a3 / 3 + a4 * 5 / 6 - a5 / 6))


def sides(f, axis, o, eps):
    n = f.shape[axis]
    at = np.arange(-3, n + 3)
    at = np.where(at < 0, 1, np.where(at >= n, n - 2, at))
    d = o * np.diff(np.take(f, at, axis), axis=axis)
    d = [np.take(d, range(k, k + n), axis) for k in range(6)]
    return weno(*d[:5], eps), weno(*d[5:0:-1], eps)


def pick(s, m, p, along_x):
    """0: m, 1: p, 2: neither, -1: phi stays (ADVECTION_METHOD_2D.h:1505-1655)."""
    sm, sp = s * m, s * p
    sss = s * (np.abs(p) - np.abs(m)) / (p - m)
    shock = np.where(sss > 0, 0, np.where((sss < 0) | (not along_x), 1, -1))
    return np.select([(sp >= 0) & (sm >= 0), (sp <= 0) & (sm <= 0), (sp > 0) & (sm < 0), (sp < 0) & (sm > 0)],
                     [0, 1, 2, shock], -1)


def sweep(phi, s, dtau, odx, ody, eps):
    f = phi[2:-2, 2:-2]
    out = phi.copy()
    with np.errstate(all="ignore"):
        (mx, px), (my, py) = sides(f, 1, odx, eps), sides(f, 0, ody, eps)
        xs, ys = pick(s, mx, px, True), pick(s, my, py, False)
        gx, gy = np.where(xs == 0, mx, px), np.where(ys == 0, my, py)
        g2 = np.where(xs == 2, 0.0, gx * gx) + np.where(ys == 2, 0.0, gy * gy)
        h = np.where((xs == 2) & (ys == 2), 0.0, np.sqrt(g2)) - 1.0
        out[2:-2, 2:-2] = np.where((xs < 0) | (ys < 0), f, f - dtau * s * h)
    return out


SIGNS = [1.0, 2.0**-100, 2.0**-101, np.nextafter(2.0**100, 0), 2.0**100, 2.0**200, 1.7e308, np.inf, np.nan, 0.0]


@pytest.mark.parametrize("size", SIGNS)
@pytest.mark.parametrize("ni,nj", [(33, 5), (64, 8), (31, 17)])
def test_sweep_equals_plain_arithmetic(gb, ni, nj, size):
    case = bubbles_case(ni, nj, seed=ni + nj)
    rng = np.random.default_rng(ni)
    phi = case["phi"] * 40000 + rng.uniform(-1e-3, 1e-3, case["phi"].shape)
    s = np.sign(phi[2:-2, 2:-2])
    s[rng.random(s.shape) < 0.5] *= size  # ordinary nodes beside them, in the same tiles
    c = gb.Context(ni, nj)
    got = c.reinit_sweep(phi, s)
    c.close()
    dx, dy = 1.0 / (ni - 1), 1.0 / (nj - 1)
    np.testing.assert_array_equal(got, sweep(phi, s, dx / 5.0, 1.0 / dx, 1.0 / dy, 1e-6))
