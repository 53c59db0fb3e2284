"""A frame formed at once (sww_frame) in between leaves the asynchronous frame
that was started last as it was: waiting for it again gives the same values,
whether its buffer was handed over or not, and when another thread waits (exact
comparisons)."""
import concurrent.futures

import numpy as np
import pytest

from anuga_core_gb300.workloads import dam_break

pytestmark = pytest.mark.gpu


def _scenario(m):
    d = dam_break(m, "DE1", precision="fp64")
    flat = d.mesh.triangles.ravel()
    off = np.zeros(d.mesh.number_of_nodes + 1, np.int64)
    off[1:] = np.cumsum(np.bincount(flat, minlength=d.mesh.number_of_nodes))
    d.advance_steps(1)
    d._scn.sww_bind(off, np.argsort(flat, kind="stable"))
    return d, d._scn


def _same(a, b):
    return np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


# waits before and after the immediate frame
@pytest.mark.parametrize("before,after", [(1, 1), (0, 1), (0, 2), (1, 2), (2, 2)])
@pytest.mark.parametrize("m", [1, 24])
def test_immediate_frame_between_waits(m, before, after):
    d, scn = _scenario(m)
    first = scn.sww_frame(1.0e-3)
    scn.sww_frame_async(1.0e-3)
    for _ in range(before):
        assert _same(scn.sww_frame_wait(), first)
    d.advance_steps(3)
    second = scn.sww_frame(1.0e-3)
    assert not np.array_equal(first[1], second[1])
    held = [scn.sww_frame_wait() for _ in range(after)]
    assert all(_same(f, first) for f in held)
    scn.sww_frame_async(1.0e-3)
    assert _same(scn.sww_frame_wait(), second) and _same(scn.sww_frame_wait(), second)
    assert all(_same(f, first) for f in held)


def test_waiting_in_another_thread():
    d, scn = _scenario(40)
    with concurrent.futures.ThreadPoolExecutor(max_workers=1) as ex:
        for _ in range(30):
            want = scn.sww_frame(1.0e-3)
            scn.sww_frame_async(1.0e-3)
            waiting = ex.submit(scn.sww_frame_wait)
            d.advance_steps(1)
            scn.sww_frame(1.0e-3)
            assert _same(waiting.result(), want)
            assert _same(scn.sww_frame_wait(), want)
