"""States that the integer fluxes leave to the FP64 forms.

Negative density: with B = 0 the flux of -Q is that of Q negated and the velocities are the same, so
the A_z advection must not change.  Tolerance: the whole-run bound of 1e-10 relative L2."""
import numpy as np
import pytest

import oracle
from chorus_mhd import Mesh, Solver, reference_layout_sizes
from helpers import assert_close, make_case

pytestmark = pytest.mark.gpu
TOL = 1e-10


@pytest.mark.parametrize("N", [2, 4, 5])
def test_negative_density_keeps_the_upwind_side(case_root, N):
    d = make_case(case_root, problem="orszag_tang", nx=9, ny=8, N=N, jitter=0.1, seed=N)
    o = oracle.Oracle(d)
    s = Solver(Mesh(d), initial_state=False)
    Q = o.array("Q").reshape(-1, 9).copy()
    Q[:, 4] -= 0.5 * (Q[:, 5:8] ** 2).sum(1)
    Q[:, 5:8] = 0.0
    Q[:, :8] *= -1
    o.array("Q")[...] = Q.reshape(o.array("Q").shape)
    s.upload(Q)
    o.compresid()
    s.compresid()
    n = reference_layout_sizes(N, s.ncell)["resid"]
    a, b = s.array("resid", n).reshape(-1, 9), o.array("resid").reshape(-1, 9)
    assert_close(a[:, 8], b[:, 8], TOL, "A_z advection")
    assert_close(a[:, :5], b[:, :5], TOL, "residual")
