"""The windows of the integer point fluxes (chorus-mhd_gb300/csrc/intflux.cuh), on the host: magnitudes
up to the windows' ends and past them.  A point that the integer form takes has a result within
the range of a double; where the FP64 form overflows, the point is refused."""
import numpy as np
import pytest

from test_intflux import LD, driver, evaluate, physics, pytestmark  # noqa: F401
from test_intflux_components import exact_flux, normals, terms

MAX = np.finfo(np.float64).max


def big(rng, shape, top):
    return rng.choice([-1.0, 1.0], shape) * 2.0 ** rng.uniform(-top, top, shape)


def viscous_terms(q, G, N, mu, eta, gam):
    """Sums of the magnitudes of the viscous flux's terms, and of its largest intermediate product."""
    q, G, N = abs(q), abs(G), abs(N)
    rho, u, B = q[:, 0], q[:, 1:4] / q[:, :1], q[:, 5:8]
    rel = G[:, :, 1:4] + G[:, :, :1] * u[:, None]
    S = N.sum(1)
    c = 4 * rel.sum((1, 2)) * S
    X = (u * u).sum(1) + (B * B).sum(1) / rho + q[:, 4] / rho
    GS = (G * N[:, :, None]).sum(1)
    heat = GS[:, 4] + (u * GS[:, 1:4]).sum(1) + (B * GS[:, 5:8]).sum(1) + X * GS[:, 0]
    return mu / rho * (c * (1 + u.sum(1)) + gam / LD(0.72) * heat) + eta * G.sum((1, 2)) * S * (1 + B.sum(1))


@pytest.mark.parametrize("top", [60, 119, 150, 199, 300])
def test_viscous_flux(driver, tmp_path, top):  # noqa: F811
    rng = np.random.default_rng(top)
    n = 4000
    q, G, N = big(rng, (n, 8), top), big(rng, (n, 2, 8), top), big(rng, (n, 2), top)
    q[:, 0] = abs(q[:, 0])
    q[: n // 4, 0] = 2.0 ** -rng.uniform(0.9 * top, top, n // 4)  # light and fast: the largest velocities
    q[: n // 4, 1:4] = 2.0 ** rng.uniform(0.9 * top, top, (n // 4, 3))
    G[: n // 4] = 2.0 ** rng.uniform(0.9 * top, top, (n // 4, 2, 8))
    mu, eta = abs(big(rng, (2, n), top))
    out = evaluate(driver, tmp_path, 2, np.concatenate([q, G.reshape(n, 16), mu[:, None], eta[:, None], N, np.full((n, 1), 5 / 3)], 1))
    took = out[:, 0] == 1
    scale = viscous_terms(*[x.astype(LD) for x in (q, G, N, mu, eta)], LD(5) / 3)
    if top <= 119:
        assert took.all()
    assert np.all(scale[took] < MAX)
    assert np.all(np.isfinite(out[took]))
    assert np.all(abs(out[took, 1:]) <= 2 * scale[took][:, None])


@pytest.mark.parametrize("top", [60, 150, 199, 300])
def test_ideal_fluxes(driver, tmp_path, top):  # noqa: F811
    """Their pressure check bounds the momentum and the field by the energy."""
    rng = np.random.default_rng(1000 + top)
    n = 4000
    q = big(rng, (n, 8), top)
    q[:, 0] = abs(q[:, 0])
    ke = ((q[:, 1:4].astype(LD) ** 2).sum(1) / q[:, 0] + (q[:, 5:8].astype(LD) ** 2).sum(1)) / 2
    fits = rng.random(n) < 0.7  # momentum and field that an energy within the window holds
    cut = np.minimum(1, np.sqrt(2.0 ** (top - 1.0) / ke)).astype(np.float64)[fits, None]
    q[fits, 1:4], q[fits, 5:8] = q[fits, 1:4] * cut, q[fits, 5:8] * cut
    ke = ((q[:, 1:4].astype(LD) ** 2).sum(1) / q[:, 0] + (q[:, 5:8].astype(LD) ** 2).sum(1)) / 2
    q[:, 4] = np.minimum((ke * 2.0 ** rng.uniform(0.01, 3, n)).astype(LD), LD(2.0) ** (top * 1.0)).astype(np.float64)
    S = big(rng, (n, 2), top)
    out = evaluate(driver, tmp_path, 1, np.concatenate([q, S, np.full((n, 1), 5 / 3)], 1))
    took = out[:, 0] == 1
    L, M, g = q.astype(LD), S.astype(LD), LD(5) / 3
    F, p, _ = exact_flux(L, M, g)
    scale = terms(L, M, g)[0]
    assert np.all(took[(p > 0) & fits & (q[:, 4] > 2.0 ** -200)]) if top < 200 else not took[abs(q).max(1) > 2.0 ** 201].any()
    assert np.all(scale[took] < MAX) and np.all(p[took] >= -abs(q[took, 4]))
    assert np.all(abs(out[took, 1:] - F[took]) <= np.maximum(LD(2.0) ** -52 * scale[took], 2.0 ** -1022))
    N = normals(rng, "any", n)
    sc = big(rng, n, top)
    out = evaluate(driver, tmp_path, 0, np.concatenate([q, q, N, sc[:, None], np.full((n, 1), 5 / 3)], 1))
    took = out[:, 0] == 1
    F, _, _ = exact_flux(L, N.astype(LD), g)
    scale = 2 * abs(sc[:, None]) * terms(L, N.astype(LD), g)[0]
    assert np.all(scale[took] < MAX)
    assert np.all(abs(out[took, 1:9] - 2 * sc[took, None] * F[took]) <= np.maximum(LD(2.0) ** -52 * scale[took], 2.0 ** -1022))
