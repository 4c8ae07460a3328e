"""The integer point fluxes (chorus-mhd_gb300/csrc/intflux.cuh) component by component: states
whose components differ by many orders of magnitude, along normals on, beside and off the axes,
against extended precision, on the host.

Tolerance: as the FP64 forms do, the integer forms keep each term of a component's sum to its own
size, so a component is held to 2^-52 of the sum of the magnitudes of its own terms (half an ulp
of the result, 2^-53, and some units of 2^-55 for the products and sums before it).  A term that
is itself a sum (the velocity along the normal, the pressure, ...) enters with the magnitudes of
that sum's terms."""
import numpy as np
import pytest

from test_intflux import LD, driver, evaluate, physics, pytestmark  # noqa: F401

EPS = LD(2.0) ** -52
GAMMAS = [1.05, 1.4, 5.0 / 3, 2.0]


def spread(rng, n, lo=-18):
    """Magnitudes from 10^lo to 1, a tenth of them zero, of either sign."""
    a = 10.0 ** rng.uniform(lo, 0, n) * rng.choice([-1.0, 1.0], n)
    a[rng.random(n) < 0.1] = 0.0
    return a


def normals(rng, kind, n):
    th = rng.uniform(0, 2 * np.pi, n)
    if kind != "any":
        th = rng.integers(0, 4, n) * (np.pi / 2)
    N = np.stack([np.cos(th), np.sin(th)], 1)
    if kind != "any":
        N = np.rint(N)
    if kind == "near axis":  # as the rounding of a mesh's vertices leaves it
        N[N == 0] = (10.0 ** rng.uniform(-20, -1, n) * rng.choice([-1, 1], n))
    return N


def exact_flux(q, n, gam):
    """physics() with the induction terms of the plane as (v Bx - u By) (ny, -nx), which does not cancel."""
    F, p, vn, _ = physics(q, n, gam)
    W = (q[:, 2] * q[:, 5] - q[:, 1] * q[:, 6]) / q[:, 0]
    F[:, 5], F[:, 6] = W * n[:, 1], -W * n[:, 0]
    return F, p, vn


STATES = ["transverse", "mixed", "planar mixed"]


def mixed(rng, kind, n, gam):
    """Conserved states, (n, 8): the plane's transverse components tiny, or every component of a
    size of its own."""
    rho, p = np.exp(rng.uniform(-2, 2, (2, n)))
    if kind == "transverse":
        a = 10.0 ** rng.uniform(-18, 0, n)
        v, B = rng.uniform(-1, 1, (2, 3, n))
        v[1], B[1] = a * v[1], a * B[1]
        v[2], B[2] = 0.0, 0.0
        p = p * 0.5
    else:
        v, B = np.stack([spread(rng, n) for _ in range(3)]), np.stack([spread(rng, n) for _ in range(3)])
        if kind == "planar mixed":
            v[2], B[2] = 0.0, 0.0
        p = p * 10.0 ** rng.uniform(-6, 0, n)
    flip = rng.random(n) < 0.5
    v[:2, flip], B[:2, flip] = v[1::-1, flip], B[1::-1, flip]
    E = p / (gam - 1) + 0.5 * rho * (v * v).sum(0) + 0.5 * (B * B).sum(0)
    return np.stack([rho, *(rho * v), E, *B], 1)


def terms(q, n, gam):
    """The sums of magnitudes of the terms of each flux component, the pressure's, the velocity's."""
    rho, m, E, B = q[:, 0], abs(q[:, 1:4]), abs(q[:, 4]), abs(q[:, 5:8])
    n = abs(n)
    v = m / rho[:, None]
    V, bn = (v[:, :2] * n).sum(1), (B[:, :2] * n).sum(1)
    b2, ke, mB = (B * B).sum(1), (m * v).sum(1), (m * B).sum(1)
    p = (gam - 1) * (E + ke / 2 + b2 / 2)
    pt = p + b2 / 2
    fm = m * V[:, None] + B * bn[:, None]
    fm[:, :2] += pt[:, None] * n
    W = v[:, 1] * B[:, 0] + v[:, 0] * B[:, 1]
    return np.stack([rho * V, *fm.T, (E + pt) * V + mB * bn / rho, W * n[:, 1], W * n[:, 0],
                     B[:, 2] * V + v[:, 2] * bn], 1), p, V


@pytest.mark.parametrize("gam", GAMMAS)
@pytest.mark.parametrize("normal", ["axis", "near axis", "any"])
@pytest.mark.parametrize("kind", STATES)
def test_interior_flux(driver, tmp_path, kind, normal, gam):  # noqa: F811
    rng = np.random.default_rng(1000 + 10 * STATES.index(kind) + len(normal) + int(100 * gam))
    n = 3000
    q = mixed(rng, kind, n, gam)
    S = normals(rng, normal, n) * np.exp(rng.uniform(-8, 8, (n, 1)))
    out = evaluate(driver, tmp_path, 1, np.concatenate([q, S, np.full((n, 1), gam)], 1))
    assert np.all(out[:, 0] == 1)
    Q, N, g = q.astype(LD), S.astype(LD), LD(gam)
    F = exact_flux(Q, N, g)[0]
    assert np.all(abs(out[:, 1:] - F) <= EPS * terms(Q, N, g)[0])
