"""The point fluxes in integer arithmetic (chorus-mhd_gb300/csrc/intflux.cuh), compiled for the
host with UndefinedBehaviorSanitizer (overflow of the 64-bit sums, shifts out of range), against
the formulas in extended precision.  CPU only.

Tolerance: the sums keep at least 56 bits relative to their largest possible term and are
rounded once, so a component is off by at most half an ulp of the result (2^-53) and a few units
of 2^-56 of the sum's scale: below 2^-52 of that scale."""
import os
import shutil
import struct
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
LD = np.longdouble
pytestmark = pytest.mark.skipif(np.finfo(LD).nmant < 63, reason="long double has no extra bits here")


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no host compiler")
    out = str(tmp_path_factory.mktemp("intflux") / "intflux_driver")
    cmd = ["g++", "-std=c++17", "-O1", "-fsanitize=undefined", "-fno-sanitize-recover=all",
           "-I", os.path.join(ROOT, "chorus-mhd_gb300", "csrc"),
           os.path.join(HERE, "intflux", "intflux_driver.cpp"), "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


def evaluate(driver, tmp_path, kind, rec):
    src, dst = str(tmp_path / "in.bin"), str(tmp_path / "out.bin")
    with open(src, "wb") as f:
        f.write(struct.pack("<2i", kind, rec.shape[0]) + np.ascontiguousarray(rec, np.float64).tobytes())
    r = subprocess.run([driver, src, dst], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    return np.fromfile(dst, np.float64).reshape(rec.shape[0], -1)


# states: 3-D fields, planar (w = B_z = 0), small and large z parts, supersonic (pressure far below
# the energy), hydrodynamic, at rest, near the ends of the accepted range
KINDS = ["general", "planar", "small z", "guide field", "supersonic", "hydro", "rest", "tiny", "huge"]


def primitives(rng, kind, n):
    """rho, p, v, B as the rows of an (8, n) array."""
    e = lambda: np.exp(rng.uniform(-2, 2, n))  # noqa: E731
    rho, p, v, B = e(), e(), rng.uniform(-1, 1, (3, n)), rng.uniform(-1, 1, (3, n))
    if kind == "planar":
        v[2], B[2] = 0.0, 0.0
    if kind == "small z":
        v[2], B[2] = v[2] * 1e-9, B[2] * 1e-7
    if kind == "guide field":
        B[:2], B[2] = B[:2] * 1e-4, B[2] * 100
    if kind == "supersonic":
        v, p = v * 30, p * 0.1
    if kind == "hydro":
        B *= 0.0
    if kind == "rest":
        v *= 0.0
    if kind in ("tiny", "huge"):  # scales that stay within 2^-200 .. 2^200 (energy and density)
        s = 1e-25 if kind == "tiny" else 1e25
        rho, p, B = rho * s, p * s, B * np.sqrt(s)
    return np.stack([rho, p, *v, *B])


def conserved(w):
    rho, p, v, B = w[0], w[1], w[2:5], w[5:8]
    E = p / (5.0 / 3 - 1) + 0.5 * rho * (v * v).sum(0) + 0.5 * (B * B).sum(0)
    return np.stack([rho, *(rho * v), E, *B], 1)


def states(rng, kind, n):
    return conserved(primitives(rng, kind, n))


def physics(q, n, gam):
    """Flux along n, the pressure, the normal velocity and the scales of the flux's sums, in long double."""
    rho, m, E, B = q[:, 0], q[:, 1:4], q[:, 4], q[:, 5:8]
    v = m / rho[:, None]
    b2, v2 = (B * B).sum(1), (v * v).sum(1)
    p = (gam - 1) * (E - rho * v2 / 2 - b2 / 2)
    pt = p + b2 / 2
    vn, bn = (v[:, :2] * n).sum(1), (B[:, :2] * n).sum(1)
    fm = m * vn[:, None] - B * bn[:, None]
    fm[:, :2] += pt[:, None] * n
    F = np.stack([rho * vn, *fm.T, (E + pt) * vn - bn * (v * B).sum(1), *(B * vn[:, None] - v * bn[:, None]).T], 1)
    s, V, b = np.sqrt((n * n).sum(1)), np.sqrt(v2), np.sqrt(b2)
    mom = s * (rho * v2 + abs(p) + b2)
    scale = np.stack([s * rho * V, mom, mom, mom, s * V * (abs(E) + abs(p) + b2), *[s * V * b] * 3], 1)
    return F, p, vn, scale


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("axis", [False, True], ids=["any normal", "axis normal"])
def test_rusanov_against_extended_precision(driver, tmp_path, kind, axis):
    rng = np.random.default_rng(len(kind) + 100 * axis)
    n, gam = 2000, 5.0 / 3
    w = primitives(rng, kind, n)
    ql, qr = conserved(w), conserved(w * (1 + np.exp(rng.uniform(-20, -1, n)) * rng.uniform(-1, 1, w.shape)))
    qr[: n // 10] = ql[: n // 10]  # both sides equal, as on a FREE face
    th = rng.integers(0, 4, n) * (np.pi / 2) if axis else rng.uniform(0, 2 * np.pi, n)
    nn = np.stack([np.cos(th), np.sin(th)], 1)
    if axis:
        nn = np.rint(nn)
    sc = rng.choice([-1, 1], n) * np.exp(rng.uniform(-8, 8, n))
    out = evaluate(driver, tmp_path, 0, np.concatenate([ql, qr, nn, sc[:, None], np.full((n, 1), gam)], 1))
    assert np.all(out[:, 0] == 1)
    L, R, N, S = (a.astype(LD) for a in (ql, qr, nn, sc))
    g = LD(gam)
    Fl, pl, vl, sl = physics(L, N, g)
    Fr, pr, vr, sr = physics(R, N, g)
    B, rho = (L[:, 5:] + R[:, 5:]) / 2, (L[:, 0] + R[:, 0]) / 2
    ca, cd, cn = g * (pl + pr) / 2 / rho, (B * B).sum(1) / rho, (B[:, :2] * N).sum(1) ** 2 / rho
    disc = (ca + cd) ** 2 - 4 * ca * cn
    cf = np.sqrt((ca + cd + np.sqrt(disc)) / 2)
    eig = abs(vl + vr) / 2 + cf
    F = S[:, None] * (Fl + Fr - eig[:, None] * (R - L))
    # a relative error of the pressure (its cancellation against the energy) enters the wave speed
    E = abs(L[:, 4]) + abs(R[:, 4])
    cond = 1 + E / (abs(pl) + abs(pr) + (B * B).sum(1)) + np.minimum((ca + cd) / np.sqrt(disc), LD(1e6))
    assert np.all(abs(out[:, 9] - eig) <= 2.0 ** -52 * cond * eig)
    jump = np.max(np.stack([abs(R - L), 0 * L]), 0)
    jump[:, 1:3] = jump[:, 1:3].max(1)[:, None]  # the components of the plane share a scale
    jump[:, 5:7] = jump[:, 5:7].max(1)[:, None]
    scale = abs(S[:, None]) * (sl + sr + eig[:, None] * jump * cond[:, None])
    assert np.all(abs(out[:, 1:9] - F) <= 2.0 ** -52 * scale)
    zero = np.zeros((n, 8), bool)
    if kind in ("planar", "hydro"):
        zero[:, 7] = True
        zero[:, 5:7] = kind == "hydro"
    assert np.all(out[:, 1:9][zero] == 0)  # what is exactly zero stays so


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("axis", [False, True], ids=["any metric", "axis metric"])
def test_interior_flux_against_extended_precision(driver, tmp_path, kind, axis):
    rng = np.random.default_rng(50 + len(kind) + 100 * axis)
    n, gam = 2000, 5.0 / 3
    q = states(rng, kind, n)
    th = rng.integers(0, 4, n) * (np.pi / 2) if axis else rng.uniform(0, 2 * np.pi, n)
    S = np.stack([np.cos(th), np.sin(th)], 1)
    S = (np.rint(S) if axis else S) * np.exp(rng.uniform(-8, 8, (n, 1)))
    out = evaluate(driver, tmp_path, 1, np.concatenate([q, S, np.full((n, 1), gam)], 1))
    assert np.all(out[:, 0] == 1)
    F, _, _, scale = physics(q.astype(LD), S.astype(LD), LD(gam))
    assert np.all(abs(out[:, 1:] - F) <= 2.0 ** -52 * scale)
    if kind in ("planar", "hydro"):
        assert np.all(out[:, 8] == 0)  # what is exactly zero stays so
    if kind == "hydro":
        assert np.all(out[:, 6:8] == 0)


def test_states_outside_the_integer_form_are_refused(driver, tmp_path):
    """Non-finite values, densities that are not positive or not normal, a density ratio above 16,
    scales beyond the window: left to the FP64 form."""
    rng = np.random.default_rng(3)
    good = np.concatenate([*[states(rng, "general", 1)[0]] * 2, [0.6, 0.8, 1.0, 5.0 / 3]])
    bad = []
    for k, vals in ((0, [0.0, -1.0, np.nan, np.inf, 5e-324, 1e300, 20 * good[0]]), (1, [np.nan, -np.inf, 1e100]),
                    (4, [np.nan, np.inf, 0.0]), (7, [np.inf]), (18, [0.0, 1e-100, 1e100])):
        for v in vals:
            r = good.copy()
            r[k] = v
            bad.append(r)
    cold = good.copy()
    cold[4] *= 0.01  # negative pressure on one side
    bad.append(cold)
    out = evaluate(driver, tmp_path, 0, np.array([good] + bad))
    assert out[0, 0] == 1 and np.all(out[1:, 0] == 0)
    # the same states at an interior point, without the density ratio and with the metric's bounds
    inner = [[*r[:8], *r[16:18], r[19]] for r in bad if r[0] != 20 * good[0] and r[18] == 1.0]
    inner += [[*good[:8], v, v, good[19]] for v in (0.0, 1e-100, 1e100, np.nan)]
    out = evaluate(driver, tmp_path, 1, np.array([[*good[:8], 0.6, 0.8, good[19]]] + inner))
    assert out[0, 0] == 1 and np.all(out[1:, 0] == 0)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("coef", ["both", "viscous", "resistive"])
def test_viscous_flux_against_extended_precision(driver, tmp_path, kind, coef):
    """The scale leaves out factors of up to four (2 du/dx, two thirds of the divergence, two
    terms to a sum): 2^-50 of it."""
    rng = np.random.default_rng(200 + len(kind) + 50 * len(coef))
    n, gam, Pr = 2000, 5.0 / 3, 0.72
    q = states(rng, kind, n)
    size = abs(q) + 0.1 * np.sqrt(q[:, :1]) * (kind not in ("tiny", "huge"))  # of the variables' gradients
    size *= np.exp(rng.uniform(-4, 2, (n, 8)))
    if kind in ("planar", "hydro"):
        size[:, [3, 7]] = 0
    if kind == "hydro":
        size[:, 5:] = 0
    G = size[:, None, :] * rng.uniform(-1, 1, (n, 2, 8))
    th = rng.uniform(0, 2 * np.pi, n)
    S = np.stack([np.cos(th), np.sin(th)], 1) * np.exp(rng.uniform(-8, 8, (n, 1)))
    mu = 1e-3 * np.exp(rng.uniform(-2, 2, (n, 1))) * (coef != "resistive")
    eta = 1e-3 * np.exp(rng.uniform(-2, 2, (n, 1))) * (coef != "viscous")
    out = evaluate(driver, tmp_path, 2, np.concatenate([q, G.reshape(n, 16), mu, eta, S, np.full((n, 1), gam)], 1))
    assert np.all(out[:, 0] == 1)
    Q, D, M, H, N = (a.astype(LD) for a in (q, G, mu[:, 0], eta[:, 0], S))
    rho, B, g = Q[:, 0], Q[:, 5:8], LD(gam)
    u = Q[:, 1:4] / rho[:, None]
    v2, b2 = (u * u).sum(1), (B * B).sum(1)
    e = (Q[:, 4] - rho * v2 / 2 - b2 / 2) / rho
    du = (D[:, :, 1:4] - D[:, :, :1] * u[:, None]) / rho[:, None, None]
    de = (D[:, :, 4] - v2[:, None] / 2 * D[:, :, 0] - rho[:, None] * (u[:, None] * du).sum(2)
          - (B[:, None] * D[:, :, 5:8]).sum(2) - D[:, :, 0] * e[:, None]) / rho[:, None]
    div = du[:, 0, 0] + du[:, 1, 1]
    txx, tyy, txy = 2 * du[:, 0, 0] - 2 * div / 3, 2 * du[:, 1, 1] - 2 * div / 3, du[:, 0, 1] + du[:, 1, 0]
    tau = M[:, None] * np.stack([txx * N[:, 0] + txy * N[:, 1], txy * N[:, 0] + tyy * N[:, 1], (du[:, :, 2] * N).sum(1)], 1)
    J = np.stack([D[:, 1, 7], -D[:, 0, 7], D[:, 0, 6] - D[:, 1, 5]], 1)
    NJ = H[:, None] * np.stack([-J[:, 2] * N[:, 1], J[:, 2] * N[:, 0], J[:, 0] * N[:, 1] - J[:, 1] * N[:, 0]], 1)
    heat = M * (g / LD(Pr)) * (de * N).sum(1)
    F = np.concatenate([0 * tau[:, :1], tau, ((u * tau).sum(1) + heat + (B * NJ).sum(1))[:, None], NJ], 1)
    s, V, b = np.sqrt((N * N).sum(1)), np.sqrt(v2), np.sqrt(b2)
    gr, gm, gz, ge, gb, gw = (a.astype(LD) for a in (size[:, 0], np.hypot(size[:, 1], size[:, 2]), size[:, 3], size[:, 4],
                                                     np.hypot(size[:, 5], size[:, 6]), size[:, 7]))
    st, sz = M / rho * (gm + gr * V) * s, M / rho * (gz + gr * abs(u[:, 2])) * s
    en = V * (st + sz) + M / rho * (g / LD(Pr)) * s * (ge + V * (gm + gz) + b * (gb + gw) + gr * (v2 + abs(Q[:, 4]) / rho)) \
        + H * s * b * (gb + gw)
    scale = np.stack([0 * s, st, st, sz, en, H * gb * s, H * gb * s, H * gw * s], 1)
    assert np.all(abs(out[:, 1:9] - F) <= 2.0 ** -50 * scale)
