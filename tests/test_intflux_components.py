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


SIDES = ["alike", "independent", "contrast"]


def right_states(rng, kind, n, ql, gam):
    """The right sides of faces: a little off the left one; any other state; the same but with the
    momentum large where the left's is small and the field the other way round."""
    if kind == "alike":
        return ql * (1 + np.exp(rng.uniform(-20, -3, n))[:, None] * rng.uniform(-0.2, 0.2, ql.shape))
    rho = ql[:, 0] * 2.0 ** rng.uniform(-2.4, 2.4, n)
    if kind == "independent":
        q = mixed(rng, "mixed", n, gam)
        q[:, 4] = np.maximum(q[:, 4], 0.6 * (q[:, 1:4] ** 2).sum(1) / rho + 0.6 * (q[:, 5:8] ** 2).sum(1) + 1e-3)
    else:
        c = 10.0 ** rng.uniform(1, 6, n)[:, None]
        q = ql.copy()
        q[:, 1:4], q[:, 5:8] = q[:, 1:4] * c, q[:, 5:8] / c
        q[:, 4] = 0.6 * (q[:, 1:4] ** 2).sum(1) / rho + 0.6 * (q[:, 5:8] ** 2).sum(1) + ql[:, 4]
    q[:, 0] = rho
    return q


@pytest.mark.parametrize("gam", GAMMAS)
@pytest.mark.parametrize("normal", ["axis", "near axis", "any"])
@pytest.mark.parametrize("sides", SIDES)
@pytest.mark.parametrize("kind", STATES)
def test_face_flux(driver, tmp_path, kind, sides, normal, gam):  # noqa: F811
    """The wave speed enters every component with its own error: the roundings of the normal
    velocities and, through the square roots, that of the pressures."""
    rng = np.random.default_rng(3000 + 10 * STATES.index(kind) + 100 * SIDES.index(sides) + len(normal) + int(100 * gam))
    n = 2000
    ql = mixed(rng, kind, n, gam)
    qr = right_states(rng, sides, n, ql, gam)
    ratio = np.maximum(ql[:, 0] / qr[:, 0], qr[:, 0] / ql[:, 0])
    N = normals(rng, normal, n)
    N = N / np.sqrt((N * N).sum(1))[:, None]
    sc = rng.choice([-1, 1], n) * np.exp(rng.uniform(-8, 8, n))
    out = evaluate(driver, tmp_path, 0, np.concatenate([ql, qr, N, sc[:, None], np.full((n, 1), gam)], 1))
    took = out[:, 0] == 1
    L, R, M, S, g = ql.astype(LD), qr.astype(LD), N.astype(LD), sc.astype(LD), LD(gam)
    (Fl, pl, vl), (Fr, pr, vr) = exact_flux(L, M, g), exact_flux(R, M, g)
    # (left to the FP64 form: a density ratio above 8, a negative pressure)
    assert np.all(took[(ratio < 7.9) & (pl > 0) & (pr > 0)])
    (tl, el, al), (tr, er, ar) = terms(L, M, g), terms(R, M, g)
    B = (L[:, 5:] + R[:, 5:]) / 2
    P, D, bn2 = g * (pl + pr), 2 * (B * B).sum(1), 2 * (B[:, :2] * M).sum(1) ** 2
    T, rs = P + D, L[:, 0] + R[:, 0]
    disc = np.maximum(T * T - 4 * P * bn2, 0)
    cf = np.sqrt((T + np.sqrt(disc)) / (2 * rs))
    eig = abs(vl + vr) / 2 + cf
    dT = EPS * (g * (el + er) + D)
    dsq = np.minimum(T * dT / np.maximum(np.sqrt(disc), LD(1e-300)), np.sqrt(T * dT))
    deig = EPS * (al + ar + eig) + (dT + dsq) / (4 * rs * cf)
    assert np.all(abs(out[:, 9] - eig)[took] <= deig[took])
    J = R - L
    F = S[:, None] * (Fl + Fr - eig[:, None] * J)
    bound = abs(S[:, None]) * (EPS * (tl + tr + eig[:, None] * abs(J)) + deig[:, None] * abs(J))
    assert np.all(abs(out[:, 1:9] - F)[took] <= bound[took])


@pytest.mark.parametrize("coef", ["both", "viscous", "resistive"])
@pytest.mark.parametrize("normal", ["axis", "near axis", "any"])
@pytest.mark.parametrize("kind", STATES)
def test_viscous_flux(driver, tmp_path, kind, normal, coef):  # noqa: F811
    """Up to twelve products and sums of 2^-55 lie one behind the other: 2^-51 of the terms."""
    rng = np.random.default_rng(5000 + 10 * STATES.index(kind) + len(normal) + 100 * len(coef))
    n, gam, Pr = 3000, 5.0 / 3, 0.72
    q = mixed(rng, kind, n, gam)
    G = np.stack([spread(rng, 16 * n, -12 if kind == "transverse" else -18)]).reshape(n, 2, 8)
    if kind == "transverse":
        i = np.where(abs(q[:, 1]) > abs(q[:, 2]), 1, 0)  # the transverse variables of the plane
        for k in (1, 5):
            G[np.arange(n), :, k + i] *= (10.0 ** rng.uniform(-18, 0, n))[:, None]
    if "mixed" != kind:
        G[:, :, [3, 7]] = 0.0
    S = normals(rng, normal, n) * np.exp(rng.uniform(-8, 8, (n, 1)))
    mu = 1e-3 * np.exp(rng.uniform(-2, 2, (n, 1))) * (coef != "resistive")
    eta = 1e-3 * np.exp(rng.uniform(-2, 2, (n, 1))) * (coef != "viscous")
    out = evaluate(driver, tmp_path, 2, np.concatenate([q, G.reshape(n, 16), mu, eta, S, np.full((n, 1), gam)], 1))
    assert np.all(out[:, 0] == 1)

    def flux(q, G, N, M, H, s):
        """The flux (s = -1: differences as they are) or the sums of its terms' magnitudes (s = 1, all inputs >= 0)."""
        rho, E, B = q[:, 0], q[:, 4], q[:, 5:8]
        u = q[:, 1:4] / rho[:, None]
        dot = lambda a, b: (a * b).sum(-1)  # noqa: E731
        rel = G[:, :, 1:4] + s * G[:, :, :1] * u[:, None]  # rho grad u
        D = (rel[:, 0, 0] + rel[:, 1, 1]) / 3
        sh = rel[:, 0, 1] + rel[:, 1, 0]
        c = np.stack([2 * (rel[:, 0, 0] + s * D) * N[:, 0] + sh * N[:, 1], sh * N[:, 0] + 2 * (rel[:, 1, 1] + s * D) * N[:, 1],
                      dot(rel[:, :, 2], N)], 1)
        X = dot(u, u) + dot(B, B) / (2 * rho) + s * E / rho
        GS = (G * N[:, :, None]).sum(1)
        heat = GS[:, 4] + s * dot(u, GS[:, 1:4]) + s * dot(B, GS[:, 5:8]) + X * GS[:, 0]
        J = H * (G[:, 0, 6] + s * G[:, 1, 5])
        F7 = H * GS[:, 7]
        energy = M / rho * (dot(u, c) + LD(gam) / LD(Pr) * heat) + J * (B[:, 1] * N[:, 0] + s * B[:, 0] * N[:, 1]) + F7 * B[:, 2]
        return np.stack([0 * rho, *(M / rho * c.T), energy, s * J * N[:, 1], J * N[:, 0], F7], 1)

    a = [x.astype(LD) for x in (q, G, S, mu[:, 0], eta[:, 0])]
    F, scale = flux(*a, -1), flux(*[abs(x) for x in a], 1)
    assert np.all(abs(out[:, 1:9] - F) <= 2 * EPS * scale)
