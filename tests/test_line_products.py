"""The products of the gradient pass (states times metric entries along a line) where the two metric
entries, or the state and the metric along a line, differ by many orders of magnitude.

Tolerance on the host: the largest product of a line is held with at least 56 bits, and a product
is off by two of its units and one of the alignment: 2^-54 of the line's largest product.  On
the GPU, gradients on cells 10^6 times as wide as high, from the flux-point values that the pass
read, against extended precision: the weights and the sums keep more bits than that, the result
is rounded once, so 2^-52 of the sum over both lines of the largest product times the weights.
Products cut at 2^-58 of the line's largest metric entry are off by 10^3 times that."""
import os
import shutil
import struct
import subprocess
from fractions import Fraction

import numpy as np
import pytest

import oracle
from chorus_mhd import meshgen

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_each_product_keeps_its_bits(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no host compiler")
    exe = str(tmp_path / "driver")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=undefined", "-fno-sanitize-recover=all", "-I",
                        os.path.join(ROOT, "chorus-mhd_gb300", "csrc"),
                        os.path.join(HERE, "fixdot", "line_products_driver.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    rng = np.random.default_rng(0)
    n = 400
    q, s = rng.uniform(-1, 1, (n, 6)), rng.uniform(-1, 1, (n, 6))
    size = 10.0 ** rng.uniform(-30, 30, (n, 6))  # large states on small entries
    q[100:200], s[100:200] = q[100:200] * size[100:200], s[100:200] / size[100:200]
    s[200:300] *= 10.0 ** rng.uniform(-25, 0, (100, 1))
    q[300:320] *= rng.random((20, 6)) < 0.5
    s[320:340] *= rng.random((20, 6)) < 0.5
    q[340], s[341] = 0.0, 0.0
    src, dst = str(tmp_path / "in.bin"), str(tmp_path / "out.bin")
    with open(src, "wb") as f:
        f.write(struct.pack("<i", n) + q.tobytes() + s.tobytes())
    r = subprocess.run([exe, src, dst], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
    out = np.fromfile(dst, np.float64).reshape(n, 13)
    for o, a, b in zip(out, q, s):
        p = [Fraction(float(x)) * Fraction(float(y)) for x, y in zip(a, b)]
        top = max(abs(x) for x in p)
        unit = Fraction(2) ** int(o[0])
        X = [int(o[1 + 2 * k]) * 2 ** 30 + int(o[2 + 2 * k]) for k in range(6)]
        assert max(abs(x) for x in X) < 2 ** 58
        for x, e in zip(X, p):
            assert abs(x * unit - e) <= top / 2 ** 54
            assert e != 0 or x == 0


class Wide(meshgen.CaseSpec):
    """Cells 10^6 times as wide as high."""

    def domain(self):
        return 0.0, 2 * np.pi, 0.0, 2e-6 * np.pi, "FREE"


@pytest.mark.gpu
@pytest.mark.parametrize("N", [2, 3, 5, 8])
def test_gradients_on_flat_cells(tmp_path, N):
    from chorus_mhd import Mesh, Solver
    d = str(tmp_path / "wide")
    meshgen.write_case(Wide(nx=6, ny=5, N=N, problem="orszag_tang", jitter=0.1, seed=3, mu=0.01, eta0=0.02, artiv=0, dt=1e-9), d)
    o = oracle.Oracle(d)
    s = Solver(Mesh(d), initial_state=False)
    NC = s.ncell
    x = o.array("XXsolu").reshape(NC, N * N, 2)
    X, Y = x[:, :, 0], x[:, :, 1] * 1e6
    Q = np.stack([2 + 0.3 * np.sin(X + k) * np.cos(Y - 2 * k) for k in range(9)], -1).reshape(-1)
    Q.reshape(-1, 9)[:, 4] += 30
    s.upload(Q)
    s.compresid()
    LD = np.longdouble
    m = s.mesh
    M = m.darray("Mmat").reshape(N, N + 1).astype(LD)  # [solution point][flux point]
    J = m.darray("Jac").reshape(NC, N, N).astype(LD)
    S1 = m.darray("S1").reshape(NC, N, N + 1, 2, 2).astype(LD)[..., :, 0]  # [cell][eta][f][d]
    S2 = m.darray("S2").reshape(NC, N + 1, N, 2, 2).astype(LD)[..., :, 1]  # [cell][f][xi][d]
    a = s.array("Qvfi", NC * N * (N + 1) * 9).reshape(NC, N, N + 1, 9)[..., :8].astype(LD)
    b = s.array("Qvfj", NC * N * (N + 1) * 9).reshape(NC, N + 1, N, 9)[..., :8].astype(LD)
    g = s.array("nablaQs", NC * N * N * 18).reshape(NC, N, N, 2, 9)[..., :8]
    W = abs(M).sum(1)
    for axis in (0, 1):
        pa, pb = a * S1[..., axis, None], b * S2[..., axis, None]
        exact = (np.einsum("if,cjfk->cjik", M, pa) + np.einsum("jf,cfik->cjik", M, pb)) / J[..., None]
        bound = (abs(pa).max(2)[:, :, None] * W[None, None, :, None] + abs(pb).max(1)[:, None] * W[None, :, None, None]) / J[..., None]
        assert np.all(abs(g[:, :, :, axis] - exact) <= LD(2.0) ** -52 * bound)
