"""The viscous work on either side of the size from which it runs in a pass of its own
(49152 solution points), over a list of scattered active cells: residual, steps, skipping and the
batched form.

Tolerance: the artificial viscosity goes through log10 and sin of a ratio of sums, so the residual
is held to the whole-run bound of 1e-10 relative L2; skipped work is an exact zero, so skipping
changes nothing; batched and alone run the same arithmetic."""
import numpy as np
import pytest

import oracle
from chorus_mhd import Batch, Mesh, Solver, reference_layout_sizes
from helpers import assert_close, make_case

pytestmark = pytest.mark.gpu
TOL = 1e-10

# (N, nx, ny): just below and just above the size, for cells per group 1 and more, odd counts
SIZES = [(2, 111, 110), (2, 111, 111), (3, 73, 74), (3, 74, 74), (4, 55, 55), (4, 56, 55), (5, 41, 47), (5, 43, 46),
         (6, 33, 42), (7, 33, 31), (8, 27, 28), (8, 28, 28)]


def noisy(Q, N, NC, share, seed):
    """The state with the density of a share of the cells, spread over the mesh, made rough
    enough for the sensor.  Q is (NC, N, N, 9) with the nine variables last."""
    rng = np.random.default_rng(seed)
    q = Q.copy().reshape(NC, N * N, 9)
    hit = rng.random(NC) < share
    q[hit, :, 0] *= 1 + 0.2 * rng.uniform(-1, 1, (hit.sum(), N * N))
    return q.reshape(Q.shape)


def spec(N, nx, ny, **kw):
    return dict(problem="orszag_tang", nx=nx, ny=ny, N=N, jitter=0.1, seed=N, **kw)


@pytest.mark.parametrize("kw", [dict(), dict(mu=0.01, eta0=0.02)], ids=["av", "viscous"])
@pytest.mark.parametrize("size", SIZES, ids=lambda s: "N%d-%dx%d" % s)
def test_residual_and_steps_match_oracle(case_root, size, kw):
    d = make_case(case_root, **spec(*size, **kw))
    o = oracle.Oracle(d)
    s = Solver(Mesh(d), initial_state=False)
    N, NC = s.N, s.ncell
    Q = noisy(o.array("Q"), N, NC, 0.03, 1)
    o.array("Q")[...] = Q
    s.upload(Q)
    o.compresid()
    s.compresid()
    if not kw:
        hot = (o.array("muAVfi").reshape(NC, 2, 9)[:, :, 0] > 0).any(1)
        assert 0 < hot.sum() < NC / 2
    assert_close(s.array("resid", reference_layout_sizes(N, NC)["resid"]), o.array("resid"), TOL, "residual")
    o.run(2)
    s.iterations(2)
    assert_close(s.state(), o.array("Q"), TOL, "Q after two steps")


@pytest.mark.parametrize("share", [0.0, 0.002, 0.05, 1.0])
@pytest.mark.parametrize("size", SIZES[2:8], ids=lambda s: "N%d-%dx%d" % s)
def test_skipping_and_batch_change_nothing(case_root, size, share):
    d = make_case(case_root, **spec(*size))
    first = Solver(Mesh(d))
    Q = noisy(first.state(), first.N, first.ncell, share, 2)
    out = []
    for skip in (1, 0):
        s = Solver(Mesh(d), initial_state=False)
        s.set_option("skip_inactive_viscous", skip)
        s.set_option("diagnostics", 0)
        s.upload(Q)
        s.iterations(3)
        out.append(s.state())
    b = Batch()
    members = [Solver(Mesh(d), initial_state=False) for _ in range(2)]
    for m, q in zip(members, (Q, first.state())):
        m.upload(q)
        b.add(m)
    b.step(3)
    b.sync()
    assert np.all(np.isfinite(out[0]))
    assert np.array_equal(out[0], out[1])
    assert np.array_equal(members[0].state(), out[0])


@pytest.mark.parametrize("N,side,epb", [(2, 200, 64), (4, 164, 42), (5, 130, 27), (8, 84, 11)])
def test_most_cells_per_cta_of_the_last_pass(case_root, N, side, epb):
    """The largest option values that fit the shared memory give the same bits as the tuned one."""
    d = make_case(case_root, **spec(N, side, side))
    out = []
    for e in (None, epb):
        s = Solver(Mesh(d))
        if e:
            s.set_option("epb_e3", e)
        s.iterations(1)
        out.append(s.state())
    assert np.array_equal(out[0], out[1])
