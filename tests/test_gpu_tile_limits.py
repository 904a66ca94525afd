"""Tiles whose dynamic shared memory is just below 48 KB, the default limit of
a block: it counts the kernel's own static arrays too.  k_dt takes 20 bytes per
row of the tile and its halo and 10 per entry; seven fans of one 32-row slice
each and one that straddles the tile's end make 49120 bytes of it (137 entry
columns with 8 halo rows, 136 with 24), or one column, 320 bytes, less and
more."""
import numpy as np
import pytest

from swe import cases as C, mesh as M
from swe.update import Update
from test_gpu_tiles import _fan, _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("k,total", [(37, 99), (37, 100), (37, 101), (52, 84), (53, 83), (54, 82), (55, 81)])
def test_tile_just_below_48_kb(monkeypatch, k, total, prec):
    rng = np.random.default_rng(total)
    items = []
    for f in [total // 7 + (q < total % 7) for q in range(7)] + [k]:
        n = f + 1
        u = np.vstack([rng.uniform(0.5, 1.0, n), rng.normal(0, 0.1, n), rng.normal(0, 0.1, n)])
        items.append(C.Case("fan", _fan(f), C.Params(max_water_h=1.0, precision=prec), rng.uniform(0.0, 0.3, n),
                            np.asfortranarray(u), 1e30))
    _same(monkeypatch, items, np.hstack([c.u0 for c in items]))


def _scattered(nx, ny, lines):
    """A lattice numbered line by line, each node moved by up to `lines` lines, and one node so far away that the
    others share a cell of the Z-order's grid, which then keeps their numbering."""
    rng = np.random.default_rng(0)
    mesh = M.jittered_mesh(nx, ny, 0.0, 1.0, 0.0, ny / nx, jitter=0.2, seed=2)
    i = np.arange(nx * ny)
    at = np.argsort(np.round(mesh["rr"][1] * (nx - 1)) + rng.uniform(0.0, lines, nx * ny), kind="stable")
    new = np.empty_like(i)
    new[at] = i
    rr = mesh["rr"][:, at].copy()
    rr[:, rr.sum(axis=0).argmax()] += 1e6
    return dict(jj=np.asfortranarray(new[mesh["jj"] - 1] + 1, np.int32), rr=np.asfortranarray(rr))


@pytest.mark.parametrize("nx,ny,lines,tiled", [(330, 70, 4.0, True), (330, 310, 3.0, True), (330, 310, 6.0, False),
                                               (330, 560, 1e-3, True), (330, 560, 4.0, False)])
def test_tiles_only_where_they_are_faster(nx, ny, lines, tiled):
    """Halos of 0.4 rows per row are the rule; meshes whose numbering is loose have up to 4.5.  Small meshes take the
    tiles all the same, larger ones the global gathers above 3.65, large ones above 2.9 (sizes for 152 SMs)."""
    mesh = _scattered(nx, ny, lines)
    n = mesh["rr"].shape[1]
    rng = np.random.default_rng(1)
    u = np.asfortranarray(np.vstack([rng.uniform(0.5, 1.0, n), rng.normal(0, 0.1, (2, n))]))
    upd = Update(mesh, np.zeros(n), C.Params(max_water_h=1.0, precision=1))
    upd.upload(u)
    upd.set_time(0.0, 1e30)
    upd.rk3_steps(1)
    assert ("/tiled" in upd.tuning) == tiled, upd.tuning
    upd.close()
