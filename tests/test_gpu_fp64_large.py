"""The one-warp FP64 row kernels of large meshes (above 128 rows per SM the
low-order sweep, above 1400 k_dt) against the oracle, bit for bit, on the
states of the small-mesh tests: small instances of a batch that a filler
instance puts above both sizes."""
from dataclasses import replace

import numpy as np
import pytest

import oracle
from swe import cases as C, lib as L, mesh as M
from swe.update import Update
from test_gpu_fp64_rows import DUMPS, STATES, _both, _state

pytestmark = pytest.mark.gpu

#: (type_test, if_alpha_limit, uneven bottom) of the batch's instances
COMBOS = [(4, 1, 0), (4, 1, 1), (4, 0, 1), (11, 1, 1), (12, 1, 0)]


@pytest.fixture(scope="module")
def batch():
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    mesh = M.jittered_mesh(17, 21, 0.0, 1.0, 0.0, 1.0, jitter=0.3, seed=5)
    nn = mesh["rr"].shape[1]
    side = int((1400 * sms) ** 0.5) + 2
    fill = M.jittered_mesh(side, side, 0.0, 1.0, 0.0, 1.0, jitter=0.0, seed=0)
    rng = np.random.default_rng(17)
    items, oracles = [], []
    for tt, alpha, bumpy in COMBOS:
        z = bumpy * rng.uniform(-0.4, 0.4, nn) * (rng.random(nn) < 0.7)
        items.append((mesh, z, C.Params(max_water_h=1.0, htiny=1e-4, type_test=tt, if_alpha_limit=alpha)))
        oracles.append(oracle.Oracle(mesh["jj"], mesh["rr"]))
        oracles[-1].set_bath(z)
    items.append((fill, np.zeros(side * side), C.Params(max_water_h=1.0)))
    upd = Update(batch=items)
    yield [p for _, _, p in items], oracles, upd, nn
    upd.close()


@pytest.mark.parametrize("k", range(len(COMBOS)))
@pytest.mark.parametrize("kind", STATES)
def test_stage_bit_exact_above_the_four_warp_sizes(batch, kind, k):
    params, oracles, upd, nn = batch
    p, o = params[k], oracles[k]
    rng = np.random.default_rng(300 + STATES.index(kind))
    for _ in range(3):
        u = _state(kind, nn, p.htiny, rng)
        o.set_params(oracle.Params(*p.fields()))
        upd.set_params(p, inst=k)
        ref, got = _both(lambda: o.compute_dij(u), lambda: upd.compute_dij(u, inst=k), (L.SWE_ERR_DELTA,))
        if ref is None:
            continue
        np.testing.assert_array_equal(got[0], ref[0])
        assert got[1] == ref[1]
        pd = replace(p, dt=ref[1])
        o.set_params(oracle.Params(*pd.fields()))
        upd.set_params(pd, inst=k)
        ref, got = _both(lambda: o.euler(u, dump=True), lambda: upd.euler(u, inst=k),
                         (L.SWE_ERR_NEG_H, L.SWE_ERR_DELTA, L.SWE_ERR_NAN))
        if ref is None:
            continue
        inter = upd.euler_intermediates(inst=k)
        for name in DUMPS:
            np.testing.assert_array_equal(inter[name], ref[1][name], err_msg=name)
        np.testing.assert_array_equal(got, ref[0])
