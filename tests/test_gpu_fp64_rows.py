"""The FP64 row kernels against the oracle, bit for bit, on states chosen to
take every branch of their wave-speed bound and of their row sums: thin films
about htiny, two dry nodes, equal and nearly equal depths, depth ratios about
(2 sqrt2 - 1)^2, strong compression and expansion, supercritical flow, depths
far outside the ordinary range.  No tolerance: the kernels form the oracle's
own roundings."""

from dataclasses import replace

import numpy as np
import pytest

import oracle
from swe import cases as C, mesh as M
from swe import lib as L
from swe.update import Update

pytestmark = pytest.mark.gpu

STATES = ["rest", "equal", "near_equal", "ratio", "film", "dry", "compress", "expand", "fast", "mixed", "tiny", "huge",
          "cliff"]


def _state(kind, n, htiny, rng):
    h = rng.uniform(0.5, 1.5, n)
    v = rng.normal(0.0, 0.3, (2, n))
    if kind == "rest":
        h[:], v[:] = 0.7, 0.0
    elif kind == "equal":
        h[:] = 0.7
    elif kind == "near_equal":
        h = 0.7 * (1.0 + rng.integers(-3, 4, n) * 2.0 ** -52)
        v *= 1e-9
    elif kind == "ratio":                        # about the two-rarefaction limit of the depth ratio
        h = np.where(rng.random(n) < 0.5, 1.0, 3.3431457505 * (1.0 + rng.uniform(-2e-4, 2e-4, n)))
    elif kind == "film":
        h = htiny * (1.0 + rng.choice([-1e-3, -1e-6, -1e-12, 0.0, 1e-12, 1e-6, 1e-3, 2.0], n))
        v *= 0.01
    elif kind == "dry":
        h = np.where(rng.random(n) < 0.6, 0.0, h)
    elif kind in ("compress", "expand"):         # |vl - vr| about 1.888 sqrt(g h)
        v = (1 if kind == "expand" else -1) * rng.normal(0.0, 6.0, (2, n))
    elif kind == "fast":
        v = np.array([[300.0], [-200.0]]) + v
    elif kind == "mixed":
        h = np.exp(rng.uniform(np.log(1e-3 * htiny), np.log(2.0), n)) * (rng.random(n) < 0.9)
        v *= np.where(h < 10 * htiny, 0.01, 1.0)
    elif kind == "tiny":
        h = np.where(rng.random(n) < 0.5, h, 10.0 ** rng.uniform(-300, -20, n))
    elif kind == "cliff":                        # depth ratios of 10 to 100, phi(x0 hmin) of both signs
        h = rng.choice([0.02, 0.2, 1.0, 2.0], n) * rng.uniform(0.9, 1.1, n)
        v *= 5.0
    elif kind == "huge":
        h = h * 1e30
        v *= 1e14
    return np.asfortranarray(np.vstack([h, h * v[0], h * v[1]]))


def _pair(mesh, bath, p):
    o = oracle.Oracle(mesh["jj"], mesh["rr"])
    o.set_params(oracle.Params(*p.fields()))
    o.set_bath(bath)
    return o, Update(mesh, bath, p)


def _both(f_oracle, f_gpu, codes):
    """The oracle's result and the GPU's, or (None, None) where both refuse."""
    try:
        ref = f_oracle()
    except oracle.OracleError:
        with pytest.raises(L.SweError) as e:
            f_gpu()
        assert e.value.code in codes
        return None, None
    return ref, f_gpu()


@pytest.mark.parametrize("n", [5, 33])
@pytest.mark.parametrize("kind", STATES)
def test_dij_bit_exact(kind, n):
    rng = np.random.default_rng(STATES.index(kind) + n)
    mesh = M.jittered_mesh(n, n, 0.0, 1.0, 0.0, 1.0, jitter=0.3, seed=4)
    p = C.Params(max_water_h=1.0, htiny=1e-4)
    o, upd = _pair(mesh, np.zeros(n * n), p)
    for _ in range(4):
        u = _state(kind, n * n, p.htiny, rng)
        ref, got = _both(lambda: o.compute_dij(u), lambda: upd.compute_dij(u), (L.SWE_ERR_DELTA,))
        if ref is not None:
            np.testing.assert_array_equal(got[0], ref[0])
            assert got[1] == ref[1]


DUMPS = ("dij_low", "muij_low", "alpha", "u_low", "res", "fctmat", "rminus", "lij")


def _normals(mesh):
    """{(i, j): c_ij / |c_ij|} of the edges, c_ij the integral of phi_i grad phi_j."""
    c = {}
    for tri in mesh["jj"].T - 1:
        a, b, d = mesh["rr"][:, tri].T
        two_area = (b[0] - a[0]) * (d[1] - a[1]) - (b[1] - a[1]) * (d[0] - a[0])
        s = np.sign(two_area)
        for k in range(3):
            p, q = mesh["rr"][:, tri[(k + 1) % 3]], mesh["rr"][:, tri[(k + 2) % 3]]
            grad = s * np.array([p[1] - q[1], q[0] - p[0]]) / 6.0         # area/3 grad phi_k
            for m in range(3):
                if m != k:
                    c[tri[m], tri[k]] = c.get((tri[m], tri[k]), 0.0) + grad
    return {e: v / np.hypot(*v) for e, v in c.items()}


@pytest.mark.parametrize("seed", [0, 1])
def test_dij_where_the_depth_limit_decides(seed):
    """Pairs of nodes whose two-rarefaction depth is cut off at x0 hmin, and
    whose larger speed is the other one without the cut."""
    rng = np.random.default_rng(seed)
    g, n = 9.81, 400_000
    x0 = (2 * np.sqrt(2.0) - 1) ** 2
    cmin = np.sqrt(g)
    ratio = rng.uniform(3.05, 3.34, n)
    swap = rng.random(n) < 0.5
    hl, hr = np.where(swap, 1.0, ratio), np.where(swap, ratio, 1.0)
    dv, mid = rng.uniform(1.75, 1.887, n) * cmin, rng.uniform(-1, 1, n) * cmin
    vl, vr = mid + dv / 2, mid - dv / 2
    hs = (dv + 2 * np.sqrt(g * hl) + 2 * np.sqrt(g * hr)) ** 2 / 16 / g

    def speeds(h):
        xl, xr = np.maximum((h - hl) / hl, 0), np.maximum((h - hr) / hr, 0)
        return (np.abs(vl - np.sqrt(g * hl) * np.sqrt((1 + xl / 2) * (1 + xl))),
                np.abs(vr + np.sqrt(g * hr) * np.sqrt((1 + xr / 2) * (1 + xr))))

    (al, ar), (tl, tr) = speeds(hs), speeds(np.minimum(x0, hs))
    pick = np.nonzero((al > 1.001 * ar) & (tr > 1.001 * tl) | (ar > 1.001 * al) & (tl > 1.001 * tr))[0]
    assert len(pick) > 50
    mesh = M.jittered_mesh(21, 21, 0.0, 10.0, 0.0, 10.0, jitter=0.3, seed=7)
    p = C.Params(max_water_h=4.0, precision=0)
    nn = mesh["rr"].shape[1]
    u = np.zeros((3, nn), order="F")
    u[0] = 1.0
    used, k = set(), 0
    for (i, j), nv in _normals(mesh).items():
        if i in used or j in used:
            continue
        used |= {i, j}
        q = pick[k % len(pick)]
        k += 1
        u[:, i] = np.r_[hl[q], hl[q] * vl[q] * nv]
        u[:, j] = np.r_[hr[q], hr[q] * vr[q] * nv]
    o, upd = _pair(mesh, np.zeros(nn), p)
    ref, got = o.compute_dij(u), upd.compute_dij(u)
    np.testing.assert_array_equal(got[0], ref[0])
    assert got[1] == ref[1]


@pytest.mark.parametrize("type_test,alpha,bumpy", [(4, 1, 0), (4, 1, 1), (4, 0, 1), (11, 1, 1), (12, 1, 0)])
@pytest.mark.parametrize("kind", STATES)
def test_fct_stage_bit_exact(kind, type_test, alpha, bumpy):
    """One 'fct' stage and its intermediates, over a flat and an uneven
    bottom, with and without alpha_limit, with the linear source terms."""
    n = 17
    rng = np.random.default_rng(100 + STATES.index(kind))
    mesh = M.jittered_mesh(n, n + 4, 0.0, 1.0, 0.0, 1.0, jitter=0.3, seed=5)
    nn = mesh["rr"].shape[1]
    z = bumpy * rng.uniform(-0.4, 0.4, nn) * (rng.random(nn) < 0.7)
    p = C.Params(max_water_h=1.0, htiny=1e-4, type_test=type_test, if_alpha_limit=alpha)
    o, upd = _pair(mesh, z, p)
    for _ in range(3):
        u = _state(kind, nn, p.htiny, rng)
        try:
            dt = o.compute_dij(u)[1]
        except oracle.OracleError:
            continue
        pd = replace(p, dt=dt)
        o.set_params(oracle.Params(*pd.fields()))
        upd.set_params(pd)
        ref, got = _both(lambda: o.euler(u, dump=True), lambda: upd.euler(u),
                         (L.SWE_ERR_NEG_H, L.SWE_ERR_DELTA, L.SWE_ERR_NAN))
        if ref is None:
            continue
        inter = upd.euler_intermediates()
        for k in DUMPS:
            np.testing.assert_array_equal(inter[k], ref[1][k], err_msg=k)
        np.testing.assert_array_equal(got, ref[0])


@pytest.mark.parametrize("visc", ["viscous", "entropy_visc"])
@pytest.mark.parametrize("kind", STATES)
def test_other_modes_bit_exact(kind, visc):
    """The same row kernels without the limiter: one stage of 'viscous'
    'type2' and of 'entropy_visc' over an uneven bottom."""
    n = 15
    rng = np.random.default_rng(200 + STATES.index(kind))
    mesh = M.jittered_mesh(n, n, 0.0, 1.0, 0.0, 1.0, jitter=0.3, seed=6)
    z = rng.uniform(-0.4, 0.4, n * n) * (rng.random(n * n) < 0.7)
    p = C.Params(max_water_h=1.0, htiny=1e-4, viscosity_type=C.VISC[visc])
    o, upd = _pair(mesh, z, p)
    for _ in range(3):
        u = _state(kind, n * n, p.htiny, rng)
        try:
            pd = replace(p, dt=o.compute_dij(u)[1])
        except oracle.OracleError:
            continue
        o.set_params(oracle.Params(*pd.fields()))
        upd.set_params(pd)
        ref, got = _both(lambda: o.euler(u), lambda: upd.euler(u),
                         (L.SWE_ERR_NEG_H, L.SWE_ERR_DELTA, L.SWE_ERR_NAN))
        if ref is not None:
            np.testing.assert_array_equal(got, ref)


@pytest.mark.parametrize("nx,ny", [(2, 2), (33, 3), (65, 64), (161, 160)])
@pytest.mark.parametrize("sgn", [0, 1])
def test_fct_steps_bit_exact(sgn, nx, ny):
    """RK3 steps of both system sizes at row counts about a warp, a block,
    several, and above the four-warp kernels' range, against the oracle."""
    if sgn:
        case = C.sgn_case(nx=max(nx, 3), ny=ny, Lx=0.01 * nx, Ly=0.01 * ny, x0=0.005 * nx, cfl=5e-4)
    else:
        mesh = M.jittered_mesh(nx, ny, 0.0, 10.0, 0.0, 10.0, jitter=0.3, seed=2)
        case = C.bump_basin_case(mesh=mesh)
        case = replace(case, params=replace(case.params, type_test=4))
    o, upd = _pair(case.mesh, case.bath, case.params)
    for comp, js, vals in case.dirichlet:
        o.set_dirichlet(comp, js, vals)
        upd.set_dirichlet(comp, js, vals)
    u, t = case.u0.copy(order="F"), 0.0
    for _ in range(9):
        t = o.rk3_step(u, t)
    upd.upload(case.u0)
    upd.set_time(0.0, 1e30)
    upd.rk3_steps(9)
    np.testing.assert_array_equal(upd.download(), u)
    assert upd.get_time()[0][0] == t


def test_mode_changes_between_calls():
    """A captured run follows a later change of the viscosity mode."""
    case = C.dam_break_case(n=21, tfinal=1.0)
    o, upd = _pair(case.mesh, case.bath, case.params)
    u, t = case.u0.copy(order="F"), 0.0
    upd.upload(case.u0)
    upd.set_time(0.0, 1e30)
    for visc in ("fct", "viscous", "entropy_visc", "fct"):
        p = replace(case.params, viscosity_type=C.VISC[visc])
        o.set_params(oracle.Params(*p.fields()))
        upd.set_params(p)
        for _ in range(3):
            t = o.rk3_step(u, t)
        upd.rk3_steps(3)
        np.testing.assert_array_equal(upd.download(), u)
