"""What a context uploads on the first use of an operator (CSR positions,
element lists and Gauss weights, gauges) is on the device when the operator's
kernels read it: the first call of many fresh contexts equals their second,
bit for bit, and the oracle's.  Sizes at which the uploads are small enough for the driver to
return before they have landed."""
from dataclasses import replace

import numpy as np
import pytest

import oracle
from swe import cases as C, mesh as M
from swe.update import Update

pytestmark = pytest.mark.gpu


def _context(n, prec, seed):
    case = C.bump_basin_case(mesh=M.jittered_mesh(n, n, 0.0, 10.0, 0.0, 10.0, jitter=0.3, seed=seed), precision=prec)
    return case, Update(case.mesh, case.bath, case.params)


@pytest.mark.parametrize("n", [3, 9, 33, 101])
def test_first_dij_is_the_oracles(n):
    for seed in range(12):
        case, upd = _context(n, 0, seed)
        o = oracle.Oracle(case.mesh["jj"], case.mesh["rr"])
        o.set_params(oracle.Params(*case.params.fields()))
        o.set_bath(case.bath)
        ref = o.compute_dij(case.u0)
        for _ in range(2):
            dij, dt = upd.compute_dij(case.u0)
            np.testing.assert_array_equal(dij, ref[0])
            assert dt == ref[1]
        upd.close()


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n", [5, 65])
def test_first_intermediates_equal_second(n, prec):
    for seed in range(6):
        case, upd = _context(n, prec, seed)
        upd.set_params(replace(case.params, dt=1e-4))
        upd.euler(case.u0)
        a, b = upd.euler_intermediates(), upd.euler_intermediates()
        for k in a:
            np.testing.assert_array_equal(a[k], b[k], err_msg=k)
        upd.close()


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n", [3, 33])
def test_first_norms_and_gauges(n, prec):
    for seed in range(6):
        case, upd = _context(n, prec, seed)
        upd.upload(case.u0)
        assert upd.norms(0) == upd.norms(0)
        upd.set_time(0.0, 1e30)
        pts = case.mesh["rr"][:, case.mesh["jj"][:, 0] - 1].mean(axis=1).reshape(2, 1)
        upd.rk3_steps(1)                           # the step is captured again when the gauges are set
        upd.set_gauges(pts)
        t, _, _ = upd.rk3_steps(1)
        times, h, _, lost = upd.read_gauges()
        assert times.shape == (1, 1) and lost == 0 and times[0, 0] == t[0]
        tri = case.mesh["jj"][:, 0] - 1
        assert abs(h[0, 0] - upd.download()[0, tri].mean()) <= 1e-12 * max(1.0, abs(h[0, 0]))
        upd.close()


@pytest.mark.parametrize("visc", ["galerkin", "viscous", "entropy_visc", "fct"])
@pytest.mark.parametrize("n", [9, 65])
def test_dij_leaves_the_intermediates_alone(n, visc):
    """euler's intermediates are those of the last euler call also after
    compute_dij on another state."""
    case, upd = _context(n, 0, 0)
    upd.set_params(replace(case.params, dt=1e-4, viscosity_type=C.VISC[visc]))
    upd.euler(case.u0)
    a = upd.euler_intermediates()
    other = case.u0.copy(order="F")
    other[0] += 0.3
    first = upd.compute_dij(other)[0]
    b = upd.euler_intermediates()
    for k in a:
        np.testing.assert_array_equal(b[k], a[k], err_msg=k)
    np.testing.assert_array_equal(upd.compute_dij(other)[0], first)
    upd.close()
