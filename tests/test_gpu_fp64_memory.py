"""The FP64 row kernels' arrays are there only where they run: a context whose
modes take the general kernels does not hold them, and gets them, with the
same results as one made so, when its modes change."""
from dataclasses import replace

import numpy as np
import pytest

from swe import cases as C, mesh as M
from swe.update import Update

pytestmark = pytest.mark.gpu


def _used(make):
    """Device memory (bytes) that make()'s context holds, and the context."""
    torch = pytest.importorskip("torch")
    free0 = torch.cuda.mem_get_info()[0]
    upd = make()
    return free0 - torch.cuda.mem_get_info()[0], upd


@pytest.mark.parametrize("sgn", [0, 1])
def test_row_arrays_only_where_they_run(sgn):
    if sgn:
        case = C.sgn_case(nx=601, ny=301, Lx=6.01, Ly=3.01, x0=3.0, cfl=5e-4)
    else:
        case = C.bump_basin_case(mesh=M.jittered_mesh(420, 420, 0.0, 10.0, 0.0, 10.0, jitter=0.3, seed=3))
    n, S = case.u0.shape[1], case.u0.shape[0]
    Update(case.mesh, case.bath, case.params).close()          # the runtime's own allocations
    pg = replace(case.params, viscosity_type=C.VISC["galerkin"])
    small, general = _used(lambda: Update(case.mesh, case.bath, pg))
    large, rows = _used(lambda: Update(case.mesh, case.bath, case.params))
    assert large - small > 0.9 * (2 * S * 8) * 5.9 * n           # the row differences alone, nearly 6 entries a node

    general.set_params(case.params)
    for upd in (general, rows):
        for comp, js, vals in case.dirichlet:
            upd.set_dirichlet(comp, js, vals)
        upd.upload(case.u0)
        upd.set_time(0.0, 1e30)
        upd.rk3_steps(2)
    np.testing.assert_array_equal(general.download(), rows.download())
    got = general.compute_dij(case.u0)
    ref = rows.compute_dij(case.u0)
    np.testing.assert_array_equal(got[0], ref[0])
    assert got[1] == ref[1]
    general.close()
    rows.close()
