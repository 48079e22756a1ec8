"""The advection adjoint against PyTorch's automatic differentiation of the same sweep in FP64
(WENO5 along each line of the ghost-filled copy, linear extrapolation into the ghost ring), at
sizes around the gather's interior rule and the block widths, on both sides of the
one-block extrapolation, with both upwind signs in every warp.  A stencil coefficient is
within 4e-12 of the sum of its line's (measured against 80-bit arithmetic on smooth, noisy and
kinked lines), hence 1e-11 of the largest value here."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def side(a, eps):
    A = [a[k] - 2 * a[k + 1] + a[k + 2] for k in range(3)]
    B = [a[0] - 4 * a[1] + 3 * a[2], a[1] - a[3], 3 * a[2] - 4 * a[3] + a[4]]
    P = [a[0] / 3 - 7 * a[1] / 6 + 11 * a[2] / 6, -a[1] / 6 + 5 * a[2] / 6 + a[3] / 3, a[2] / 3 + 5 * a[3] / 6 - a[4] / 6]
    al = [c / (eps + 13.0 / 12.0 * x * x + 0.25 * y * y) ** 2 for c, x, y in zip((0.1, 0.6, 0.3), A, B)]
    return sum(w * p for w, p in zip(al, P)) / sum(al)


def derivative(f, vel, h, eps):
    """Upwind derivative along the last axis."""
    n = f.shape[-1]
    k = np.arange(-3, n + 3)
    g = f[..., np.where(k < 0, 1, np.where(k >= n, n - 2, k))]
    d = (g[..., 1:] - g[..., :-1]) / h
    a = [d[..., m:m + n] for m in range(6)]
    return torch.where(vel > 0, side(a[:5], eps), side(a[:0:-1], eps))


def sweep(phi, ua, va, dt, dx, dy, eps):
    f = phi[2:-2, 2:-2]
    u = 0.5 * (ua[3:-3, 3:-3][:, 1:] + ua[3:-3, 3:-3][:, :-1])
    v = 0.5 * (va[3:-3, 3:-3][1:] + va[3:-3, 3:-3][:-1])
    new = f - dt * (u * derivative(f, u, dx, eps) + v * derivative(f.T, v.T, dy, eps).T)
    old_l, old_b = phi[2:-2, 1], phi[1, 2:-2]
    r0 = 2 * new[:, -1] - new[:, -2]
    r1 = 2 * r0 - new[:, -1]
    t0 = 2 * new[-1] - new[-2]
    t1 = 2 * t0 - new[-1]
    return [new, r0, r1, 2 * new[:, 0] - new[:, 1], 2 * old_l - new[:, 0], t0, t1, 2 * new[0] - new[1], 2 * old_b - new[0]]


@pytest.mark.parametrize("ni,nj", [(7, 7), (8, 9), (63, 12), (64, 65), (65, 10), (130, 33), (9, 130), (1030, 8), (8, 1030)])
@pytest.mark.parametrize("velocity", [True, False])
def test_matches_automatic_differentiation(gb, ni, nj, velocity):
    rng = np.random.default_rng(ni + 7 * nj)
    xm, ym = 1.0, (nj - 1) / (ni - 1)
    h = 1.0 / (ni - 1)
    phi = np.abs(rng.uniform(-2, 2, (nj + 4, ni + 4)) * h + np.arange(ni + 4) * h - 0.4)
    ua, va, lam = (rng.standard_normal(s) for s in ((nj + 6, ni + 7), (nj + 7, ni + 6), phi.shape))
    dt = 0.5 * h
    c = gb.Context(ni, nj, x_max=xm, y_max=ym)
    for f, a in ((gb.FIELD_PHI, phi), (gb.FIELD_UA, ua), (gb.FIELD_VA, va)):
        c.set(f, a)
    got = c.weno5_adjoint(dt, lam, velocity=velocity)
    eps = 1e-6
    c.close()
    P, U, V = (torch.tensor(a, requires_grad=True) for a in (phi, ua, va))
    L = torch.tensor(lam)
    I = L[2:-2, 2:-2]
    cots = [I, L[2:-2, -2], L[2:-2, -1], L[2:-2, 1], L[2:-2, 0], L[-2, 2:-2], L[-1, 2:-2], L[1, 2:-2], L[0, 2:-2]]
    total = sum((o * w).sum() for o, w in zip(sweep(P, U, V, dt, h, h, eps), cots))
    corners = torch.zeros_like(L)
    for j in (slice(0, 2), slice(-2, None)):
        for i in (slice(0, 2), slice(-2, None)):
            corners[j, i] = 1
    total = total + (P * L * corners).sum()
    total.backward()
    for g, w in zip(got, (P.grad, U.grad, V.grad)):
        if g is None:
            assert not velocity
            continue
        w = w.numpy()
        assert np.abs(g - w).max() <= 1e-11 * np.abs(w).max()
