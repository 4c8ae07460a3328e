"""The wave speed of the integer Rusanov flux (chorus-mhd_gb300/csrc/intflux.cuh) where the field
reverses across a face, so that the averaged field of the speed is far smaller than either side's:
against extended precision, on the host.

Tolerance: the sums of the speed keep 2^-55 of their largest term, so the pressures are off by
that share of the energies, T = gamma (pl + pr) + 2 |B|^2 by E/T of that relative to itself, the
square root of the discriminant by T / sqrt(disc) more, and the fluxes by the speed's error times
the jump.  2^-52 of these covers the roundings of the results too."""
import numpy as np
import pytest

from test_intflux import LD, conserved, driver, evaluate, physics, pytestmark  # noqa: F401


def reversed_faces(rng, n, beta, residual, gam):
    rho = np.exp(rng.uniform(-1, 1, n))
    v, B = rng.uniform(-1, 1, (3, n)), rng.uniform(-1, 1, (3, n))
    v[2] *= rng.random(n) < 0.5
    B[2] *= rng.random(n) < 0.5
    p = beta * (B * B).sum(0) / 2
    wr = [rho * np.exp(rng.uniform(-1, 1, n)), p * np.exp(rng.uniform(-1, 1, n)),
          *(v + 0.1 * rng.uniform(-1, 1, (3, n))), *(-B * (1 + residual * rng.uniform(-1, 1, (3, n))))]

    def state(w):
        w = np.stack(w)
        q = conserved(w)
        q[:, 4] += w[1] * (1 / (gam - 1) - 1 / (5.0 / 3 - 1))
        return q

    return state([rho, p, *v, *B]), state(wr)


@pytest.mark.parametrize("residual", [1e-2, 1e-4, 0.0])
@pytest.mark.parametrize("beta", [1e-2, 1e-4, 1e-6, 1e-8])
@pytest.mark.parametrize("gam", [1.05, 1.4, 5.0 / 3, 2.0])
def test_reversed_field(driver, tmp_path, beta, residual, gam):  # noqa: F811
    rng = np.random.default_rng(int(1e4 * gam) + int(-np.log10(beta)) + (17 if residual == 1e-4 else 0 if residual else 31))
    n = 4000
    ql, qr = reversed_faces(rng, n, beta, residual, gam)
    th = rng.uniform(0, 2 * np.pi, n)
    N = np.stack([np.cos(th), np.sin(th)], 1)
    out = evaluate(driver, tmp_path, 0, np.concatenate([ql, qr, N, np.ones((n, 1)), np.full((n, 1), gam)], 1))
    took = out[:, 0] == 1  # (a pressure that rounds below zero is left to the FP64 form)
    assert took.mean() > 0.9
    L, R, N, g = ql.astype(LD), qr.astype(LD), N.astype(LD), LD(gam)
    Fl, pl, vl, sl = physics(L, N, g)
    Fr, pr, vr, sr = physics(R, N, g)
    B = (L[:, 5:] + R[:, 5:]) / 2
    P, D, bn2 = g * (pl + pr), 2 * (B * B).sum(1), 2 * (B[:, :2] * N).sum(1) ** 2
    T, rs = P + D, L[:, 0] + R[:, 0]
    disc = np.maximum(T * T - 4 * P * bn2, 0)
    cf2 = (T + np.sqrt(disc)) / (2 * rs)
    eig = abs(vl + vr) / 2 + np.sqrt(cf2)
    E = L[:, 4] + R[:, 4]
    eps = LD(2.0) ** -52
    # the error of sqrt(disc) is at most that of disc over it, and the square root of that of disc
    dT = eps * E
    dsq = np.minimum(T * dT / np.maximum(np.sqrt(disc), LD(1e-300)), np.sqrt(T * dT))
    V = np.sqrt((L[:, 1:3] ** 2).sum(1)) / L[:, 0] + np.sqrt((R[:, 1:3] ** 2).sum(1)) / R[:, 0]
    deig = eps * (V + eig) + (dT + dsq) / (4 * rs * np.sqrt(cf2))
    assert np.all(abs(out[:, 9] - eig)[took] <= deig[took])
    J = abs(R - L)
    mom = np.maximum(J[:, 1], J[:, 2])
    J[:, 1], J[:, 2] = mom, mom
    F = Fl + Fr - eig[:, None] * (R - L)
    scale = eps * (sl + sr + eig[:, None] * J) + deig[:, None] * J
    assert np.all(abs(out[:, 1:9] - F)[took] <= scale[took])
