"""The work arrays after the timed stages of chorus_gpu_profile_stage are those of an evaluation at the
state that it leaves, on either side of the size from which the viscous flux takes the inviscid
one's place in the stages between: compresid on the same state gives the same bits."""
import numpy as np
import pytest

from chorus_mhd import Mesh, Solver, reference_layout_sizes
from helpers import make_case

pytestmark = pytest.mark.gpu
NAMES = ["resid", "F1", "G2", "Qvfi", "Azfi", "nablaQs", "nablaAs", "muAVfi", "muAVfj"]


@pytest.mark.parametrize("mu", [0.0, 0.01])
@pytest.mark.parametrize("N,nx,ny", [(3, 73, 74), (4, 56, 55), (5, 43, 46)])
def test_arrays_after_profiling(case_root, N, nx, ny, mu):
    s = Solver(Mesh(make_case(case_root, problem="orszag_tang", nx=nx, ny=ny, N=N, jitter=0.1, seed=N, mu=mu)))
    Q = s.state().reshape(nx * ny, -1, 9)
    Q[::7, :, 0] *= 1 + 0.2 * np.random.default_rng(N).uniform(-1, 1, Q[::7, :, 0].shape)
    s.upload(Q)
    s.profile_stage(2)
    sizes = reference_layout_sizes(N, s.ncell)
    after = {k: s.array(k, sizes[k]) for k in NAMES}
    s.compresid()
    for k in NAMES:
        assert np.array_equal(after[k], s.array(k, sizes[k])), k
