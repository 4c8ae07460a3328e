"""Device memory of the total fluxes, which only the viscous pass of meshes from 49152 solution points
on writes: a solve holds them when it can have a viscous flux of that size, and comes to hold them
when its parameters change so."""
import numpy as np
import pytest

from chorus_mhd import Mesh, Solver, _lib
from helpers import make_case

N = 4
SMALL, LARGE = (55, 55), (56, 55)  # 48400 and 49280 solution points


def mesh(root, size, **kw):
    return Mesh(make_case(root, problem="orszag_tang", nx=size[0], ny=size[1], N=N, jitter=0.1, seed=1, **kw))


def total_flux(size):
    return size[0] * size[1] * 2 * (N + 1) * N * 8 * 8


def test_only_solves_that_use_them_are_charged(case_root):
    def need(*a, **kw):
        m = mesh(case_root, *a, **kw)
        return _lib.load().chorus_mesh_device_bytes(m._h)

    for kw in (dict(), dict(artiv=0, mu=0.01), dict(artiv=0, eta0=0.01)):
        assert need(SMALL, **kw) == need(SMALL, artiv=0)
        assert need(LARGE, **kw) == need(LARGE, artiv=0) + total_flux(LARGE)
    # a cell of the small mesh takes what a cell of the large one without viscosity does (to the
    # rounding of some thirty arrays to 256 bytes)
    per = lambda size: need(size, artiv=0) / (size[0] * size[1])  # noqa: E731
    assert abs(per(SMALL) - per(LARGE)) < 30 * 256 / (55 * 55) + 1


@pytest.mark.gpu
def test_viscosity_switched_on_later(case_root):
    a = Solver(mesh(case_root, LARGE, artiv=0))
    b = Solver(mesh(case_root, LARGE, artiv=0, mu=0.01, eta0=0.02))
    assert b.device_bytes() == a.device_bytes() + total_flux(LARGE)
    Q = a.state()
    a.set_option("skip_inactive_viscous", 0)  # gradients of every cell, no viscous flux
    a.iterations(1)
    inviscid = a.state()
    plain = Solver(mesh(case_root, LARGE, artiv=0))
    plain.iterations(1)
    assert np.array_equal(plain.state(), inviscid)
    a.set_params(mu=0.01, eta0=0.02)
    assert a.device_bytes() == b.device_bytes()
    for s in (a, b):
        s.upload(Q)
        s.iterations(2)
    assert not np.array_equal(a.state(), inviscid)
    assert np.array_equal(a.state(), b.state())
