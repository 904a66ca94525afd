"""Host arrays that results are copied to (pages not mapped yet, at any
8-byte offset, already written, page-locked), and the page-locked slots that
contexts read their status back through."""
import mmap
import time

import numpy as np
import pytest

from swe import cases as C, mesh as M
from swe.update import Update

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("shift", [0, 1, 511])
def test_fresh_and_written_targets_get_the_same(prec, shift):
    """A result of 1 MB into fresh pages, into written ones and into
    page-locked memory; the bytes about it stay."""
    torch = pytest.importorskip("torch")
    case = C.bump_basin_case(mesh=M.jittered_mesh(210, 210, 0.0, 10.0, 0.0, 10.0, jitter=0.3, seed=3), precision=prec)
    upd = Update(case.mesh, case.bath, case.params)
    upd.upload(case.u0)
    ref = upd.download().ravel(order="F")
    n = ref.size
    total = n + shift + 1024
    fresh = np.frombuffer(mmap.mmap(-1, 8 * total, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS), np.float64)
    written = np.full(total, -3.0)
    pinned = torch.full((total,), -3.0, dtype=torch.float64).pin_memory().numpy()
    for buf, about in ((fresh, 0.0), (written, -3.0), (pinned, -3.0)):
        upd.download_ptr(buf.ctypes.data + 8 * shift)
        np.testing.assert_array_equal(buf[shift:shift + n], ref)
        assert (buf[:shift] == about).all() and (buf[shift + n:] == about).all()
        upd.rk3_steps_host_ptr(0, buf.ctypes.data + 8 * shift, 0)
        np.testing.assert_array_equal(buf[shift:shift + n], ref)
    upd.close()


def test_fresh_target_costs_no_more_than_mapping_it():
    """A download into a fresh array of 48 MB against filling a fresh one on
    the host, which is the mapping of its pages (both about 2 ms; one page at a
    time by reading and writing it back took 15)."""
    case = C.dam_break_case(n=1420, tfinal=1.0)
    upd = Update(case.mesh, case.bath, case.params)
    upd.upload(case.u0)
    size = case.u0.nbytes
    fill, down = [], []
    for _ in range(9):
        m = np.frombuffer(mmap.mmap(-1, size, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS), np.uint8)
        t = time.perf_counter()
        m[:] = 1
        fill.append(time.perf_counter() - t)
        m = np.frombuffer(mmap.mmap(-1, size, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS), np.uint8)
        t = time.perf_counter()
        upd.download_ptr(m.ctypes.data)
        down.append(time.perf_counter() - t)
    assert min(down) < 4.0 * min(fill), (min(down), min(fill))
    upd.close()


def test_more_contexts_than_slots():
    """70 contexts at once, batches whose status exceeds one slot among them,
    closed in another order than they were made, twice."""
    case = C.dam_break_case(n=9, tfinal=1.0)
    one = Update(case.mesh, case.bath, case.params)
    one.upload(case.u0)
    one.set_time(0.0, 1e30)
    t1, dt1, _ = one.rk3_steps(3)
    ref = one.download()
    for _ in range(2):
        many = [Update(batch=[(case.mesh, case.bath, case.params)] * (40 if k % 23 == 5 else 1)) for k in range(70)]
        for upd in many:
            upd.upload(np.hstack([case.u0] * upd.n_inst))
            upd.set_time(0.0, 1e30)
        for upd in many[::-1]:
            t, dt, _ = upd.rk3_steps(3)
            assert (t == t1[0]).all() and (dt == dt1[0]).all()
            np.testing.assert_array_equal(upd.download(), np.hstack([ref] * upd.n_inst))
        for upd in many[1::2] + many[::2]:
            upd.close()
    one.close()
