"""States that the integer fluxes leave to the FP64 forms.

Negative density: with B = 0 the flux of -Q is that of Q negated and the velocities are the same, so
the A_z advection must not change.  Tolerance: the whole-run bound of 1e-10 relative L2.

A cell of NaNs: it and its face neighbours, which have a viscosity on the face between, lose their
residuals; the next cells have no viscosity and keep theirs, with the skipping of viscous work on or
off (then every cell goes through the viscous pass), to the bit."""
import numpy as np
import pytest

import oracle
from chorus_mhd import ChorusError, Mesh, Solver, reference_layout_sizes
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


@pytest.mark.parametrize("N,nx,ny", [(2, 111, 111), (3, 74, 74), (4, 55, 55), (4, 56, 55), (5, 43, 46), (8, 28, 28)])
def test_a_cell_of_nans_stays_among_its_neighbours(case_root, N, nx, ny):
    d = make_case(case_root, problem="orszag_tang", nx=nx, ny=ny, N=N, jitter=0.1, seed=N)
    n = reference_layout_sizes(N, nx * ny)["resid"]
    bad = (ny // 2) * nx + nx // 2
    near = {bad, bad - 1, bad + 1, bad - nx, bad + nx}
    o = oracle.Oracle(d)
    Q = o.array("Q").copy().reshape(nx * ny, -1)
    Q[bad] = np.nan
    out = []
    for skip in (1, 0):
        s = Solver(Mesh(d), initial_state=False)
        s.set_option("skip_inactive_viscous", skip)
        s.upload(Q)
        with pytest.raises(ChorusError):
            s.compresid()
        out.append(s.array("resid", n).reshape(nx * ny, -1))
    lost = np.where(~np.isfinite(out[0]).all(1))[0]
    assert bad in lost and set(lost) <= near
    assert np.array_equal(out[0], out[1], equal_nan=True)
