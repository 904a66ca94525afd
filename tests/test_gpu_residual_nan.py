"""A residual that is not a number (0/0: a row at rest with max_water_h = 0,
where the rescaling of update.f90:866 is 0) reaches the state of the rows that
take it from a neighbour and ends the call, in the FP64 row kernels as in the
general ones, which a batch with a 'galerkin' instance runs."""
import ctypes

import numpy as np
import pytest

import oracle
from swe import cases as C, lib as L, mesh as M
from swe.update import Update

pytestmark = pytest.mark.gpu


def _euler(upd, u):
    """Status and result of one stage of instance 0."""
    u = np.asfortranarray(u)
    out = np.zeros_like(u, order="F")
    rc = upd._L.swe_euler(upd.h, 0, L.dp(u), L.dp(out))
    return rc, out


def _scene(kind, sgn, nx, ny):
    """u (S, np): a lake at rest, one whose left part moves, one with a dry part."""
    mesh = M.jittered_mesh(nx, ny, 0.0, 1.0, 0.0, 1.0, jitter=0.3, seed=8)
    x = mesh["rr"][0]
    h = np.full(x.size, 0.7)
    if kind == "part":
        h = np.where(x < 0.4, 0.9, 0.7)
    elif kind == "dry":
        h = np.where(x < 0.4, 0.0, 0.7)
    u = np.zeros((5 if sgn else 3, x.size))
    u[0] = h
    if sgn:
        u[3] = h * h
    return mesh, np.asfortranarray(u)


@pytest.mark.parametrize("visc", ["fct", "entropy_visc"])
@pytest.mark.parametrize("kind,sgn,nx,ny", [("rest", 0, 9, 11), ("part", 0, 17, 17), ("dry", 0, 17, 17),
                                            ("part", 0, 161, 140), ("rest", 1, 9, 11), ("part", 1, 17, 17),
                                            ("part", 1, 161, 101)])
def test_nan_residual(visc, kind, sgn, nx, ny):
    mesh, u = _scene(kind, sgn, nx, ny)
    z = np.zeros(u.shape[1])
    kw = dict(type_test=13, syst_size=5, lambda_sgn=1.0) if sgn else dict(type_test=4)
    p = C.Params(max_water_h=0.0, htiny=1e-4, dt=1e-5, viscosity_type=C.VISC[visc], **kw)
    rows = Update(mesh, z, p)
    tiny = M.jittered_mesh(3, 3, 0.0, 1.0, 0.0, 1.0, jitter=0.0, seed=0)
    general = Update(batch=[(mesh, z, p), (tiny, np.zeros(9), C.Params(**{**p.__dict__, "viscosity_type": 0}))])
    rc, got = _euler(rows, u)
    rc0, ref = _euler(general, u)
    assert rc0 == L.SWE_ERR_NAN
    assert rc == rc0
    np.testing.assert_array_equal(got, ref)

    if not sgn:
        o = oracle.Oracle(mesh["jj"], mesh["rr"])
        o.set_params(oracle.Params(*p.fields()))
        o.set_bath(z)
        assert not np.isfinite(o.euler(u)).all()


@pytest.mark.parametrize("dry", ["first", "other"])
def test_dt_of_a_nan_wave_speed(dry):
    """htiny = 0 and a dry node: 1/h is 0/0 there, and so is d_ii of its wet
    neighbours.  The dt is a NaN where node 1, with which the maximum begins, is
    one of them, and passes over the others."""
    mesh, u = _scene("rest", 0, 9, 11)
    z = np.zeros(u.shape[1])
    tri = mesh["jj"][:, (mesh["jj"] == 1).any(axis=0)][:, 0]
    u[0, tri[tri != 1][0] - 1 if dry == "first" else u.shape[1] // 2] = 0.0
    p = C.Params(max_water_h=1.0, htiny=0.0)
    o = oracle.Oracle(mesh["jj"], mesh["rr"])
    o.set_params(oracle.Params(*p.fields()))
    o.set_bath(z)
    ref = o.compute_dij(u)
    assert np.isnan(ref[1]) == (dry == "first")
    upd = Update(mesh, z, p)
    dij, dt = upd.compute_dij(u)
    np.testing.assert_array_equal(dij, ref[0])
    np.testing.assert_array_equal(dt, ref[1])
    only = ctypes.c_double()
    assert upd._L.swe_compute_dij(upd.h, 0, L.dp(np.asfortranarray(u)), None, ctypes.byref(only)) == L.SWE_OK
    np.testing.assert_array_equal(only.value, ref[1])
