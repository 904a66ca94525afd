"""The row-tile kernels of the mixed path against its global-gather kernels,
bit for bit: every launch variant performs the same IEEE operations, so no
tolerance.  Sizes about a tile (256 rows) and its remainders, rows of 2 to 80
entries, both system sizes, every viscosity mode, batches whose tiles straddle
instances, both precisions."""
from dataclasses import replace

import numpy as np
import pytest

from swe import cases as C, mesh as M
from swe.update import Update

pytestmark = pytest.mark.gpu


def _fan(k):
    """k triangles about one node: a row of k entries."""
    a = np.linspace(0.0, 2 * np.pi, k, endpoint=False)
    rr = np.vstack([np.r_[0.0, np.cos(a)], np.r_[0.0, np.sin(a)]])
    i = np.arange(k)
    jj = np.vstack([np.ones(k, int), i + 2, (i + 1) % k + 2]).astype(np.int32)
    return dict(jj=np.asfortranarray(jj), rr=np.asfortranarray(rr))


def _case(kind, nx, ny, prec, visc):
    if kind == "sgn":
        c = C.sgn_case(nx=nx, ny=ny, Lx=0.01 * nx, Ly=0.01 * ny, x0=0.005 * nx, cfl=5e-4, precision=prec)
    elif kind == "basin":
        c = C.bump_basin_case(mesh=M.jittered_mesh(nx, ny, 0.0, 10.0, 0.0, 10.0, jitter=0.3, seed=7), precision=prec)
    elif kind == "film":
        c = C.thacker_case(M.jittered_mesh(nx, ny, 0.0, 4.0, 0.0, 4.0, jitter=0.3, seed=7), precision=prec)
    else:
        c = C.dam_break_case(n=max(nx, ny), precision=prec)
    return replace(c, params=replace(c.params, viscosity_type=C.VISC[visc]))


def _run(monkeypatch, tiled, items, u0, steps):
    """The state and dt after steps RK3 steps, and one Euler stage of instance
    0, in the tile (tiled = 1) or global-gather variants."""
    monkeypatch.setenv("SWE_TILED", tiled)
    upd = Update(batch=[(c.mesh, c.bath, c.params) for c in items])
    for b, c in enumerate(items):
        for comp, js, vals in c.dirichlet:
            upd.set_dirichlet(comp, js, vals, inst=b)
    upd.upload(u0)
    upd.set_time(0.0, 1e30)
    _, dt, _ = upd.rk3_steps(steps)
    assert ("/tiled" in upd.tuning) == (tiled == "1"), upd.tuning
    u = upd.download()
    upd.set_params(replace(items[0].params, dt=float(dt[0])))
    e = upd.euler(u[:, :upd.np_[0]])
    upd.close()
    return u, dt, e


def _same(monkeypatch, items, u0, steps=9):
    a, b = (_run(monkeypatch, t, items, u0, steps) for t in ("0", "1"))
    for x, y in zip(a, b):
        np.testing.assert_array_equal(y, x)


@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("kind,nx,ny", [("basin", 16, 16), ("basin", 17, 16), ("basin", 40, 33), ("film", 25, 31),
                                        ("dam", 2, 2), ("dam", 51, 51), ("sgn", 86, 3), ("sgn", 64, 4), ("sgn", 129, 9)])
def test_fct(monkeypatch, kind, nx, ny, prec):
    c = _case(kind, nx, ny, prec, "fct")
    _same(monkeypatch, [c], c.u0)


@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("roundoff,alpha", [(1, 1), (0, 1), (1, 0)])
@pytest.mark.parametrize("kind,visc", [("dam", "galerkin"), ("dam", "viscous"), ("dam", "entropy_visc"), ("dam", "fct"),
                                       ("sgn", "viscous"), ("sgn", "entropy_visc")])
def test_modes(monkeypatch, kind, visc, roundoff, alpha, prec):
    c = _case(kind, 41, 12, prec, visc)
    c = replace(c, params=replace(c.params, if_roundoff_fix=roundoff, if_alpha_limit=alpha))
    _same(monkeypatch, [c], c.u0, steps=3)


@pytest.mark.parametrize("k", [8, 80])
def test_long_rows(monkeypatch, k):
    mesh = _fan(k)
    n = k + 1
    p = C.Params(max_water_h=1.0, precision=1)
    rng = np.random.default_rng(k)
    u0 = np.asfortranarray(np.vstack([rng.uniform(0.5, 1.0, n), rng.normal(0, 0.1, n), rng.normal(0, 0.1, n)]))
    _same(monkeypatch, [C.Case("fan", mesh, p, rng.uniform(0.0, 0.3, n), u0, 1e30)], u0)


@pytest.mark.parametrize("prec", [1, 2])
def test_tiles_straddling_instances(monkeypatch, prec):
    """Row ranges are padded to 32 rows only: a tile holds rows of several
    instances, each with its own depth scale, friction and dt."""
    items = C.batch_instances(n_inst=7, nmin=20, nmax=900, seed=5, precision=prec)
    _same(monkeypatch, items, np.hstack([c.u0 for c in items]))


@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("kind", ["basin", "sgn"])
def test_batch_above_the_size_rules(kind, prec):
    """Meshes above four 256-row blocks per SM take another turn between steps,
    and their stage 1 forms the wave speeds k_dt keeps on smaller ones; above
    1400 rows per SM the FP64 k_dt gives a slice one warp instead of four.  A
    batch above those sizes equals its instances, each below them, bit for
    bit."""
    c = _case(kind, 340, 330, prec, "fct")
    one = Update(c.mesh, c.bath, c.params)
    one.upload(c.u0)
    one.set_time(0.0, 1e30)
    _, dt1, _ = one.rk3_steps(3)
    u1 = one.download()
    one.close()
    both = Update(batch=[(c.mesh, c.bath, c.params)] * 2)
    both.upload(np.hstack([c.u0, c.u0]))
    both.set_time(0.0, 1e30)
    _, dt2, _ = both.rk3_steps(3)
    u2 = both.download()
    both.close()
    n = u1.shape[1]
    assert n < 4 * 256 * 152 < 1400 * 152 < 2 * n
    for b in (0, 1):
        np.testing.assert_array_equal(u2[:, b * n:(b + 1) * n], u1)
        assert dt2[b] == dt1[0]
