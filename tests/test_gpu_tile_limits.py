"""Tiles whose dynamic shared memory is just below 48 KB, the default limit of
a block: it counts the kernel's own static arrays too.  k_dt takes 20 bytes per
row of the tile and its halo and 10 per entry; seven fans of one 32-row slice
each and one that straddles the tile's end make 49120 bytes of it (137 entry
columns with 8 halo rows, 136 with 24), or one column, 320 bytes, less and
more."""
import numpy as np
import pytest

from swe import cases as C
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
