"""Output frames are the caller's own: a frame kept while the run goes on
stays as it was, a second wait gives the same frame, and frames outlive their
scenario (both forms, exact comparisons of what the device wrote)."""
import gc

import numpy as np
import pytest

from anuga_core_gb300.batch import Batch
from anuga_core_gb300.workloads import dam_break

pytestmark = pytest.mark.gpu


def _bind(mesh):
    flat = mesh.triangles.ravel()
    off = np.zeros(mesh.number_of_nodes + 1, np.int64)
    off[1:] = np.cumsum(np.bincount(flat, minlength=mesh.number_of_nodes))
    return off, np.argsort(flat, kind="stable")


def _frames(form, m):
    """(advance and frame, wait again, close) of a dam break of 4 m^2 triangles."""
    d = dam_break(m, "DE1", precision="fp64" if form == "plain" else "mixed")
    off, slots = _bind(d.mesh)
    P = d.mesh.number_of_nodes
    if form == "plain":
        d.advance_steps(1)
        scn = d._scn
        scn.sww_bind(off, slots)

        def frame():
            d.advance_steps(2)
            scn.sww_frame_async(1.0e-3)
            return scn.sww_frame_wait()
        return frame, scn.sww_frame_wait, scn.close
    b = Batch([d])
    b.pool.sww_bind(b.sids[0], off, slots)

    def frame():
        b.advance_steps(2)
        b.pool.sww_frame_async(b.sids[0], 1.0e-3)
        return b.pool.sww_frame_wait(b.sids[0], P)
    return frame, lambda: b.pool.sww_frame_wait(b.sids[0], P), b.close


@pytest.mark.parametrize("m", [1, 24, 60])
@pytest.mark.parametrize("form", ["plain", "mixed"])
def test_frames_are_the_callers_own(form, m):
    frame, again, close = _frames(form, m)
    v, c = frame()
    v2, c2 = again()
    assert np.array_equal(v, v2) and np.array_equal(c, c2)
    assert not np.shares_memory(c, c2)
    kept_v, kept_c = v.copy(), c.copy()
    del v2, c2
    held = [frame() for _ in range(4)]
    assert np.array_equal(v, kept_v) and np.array_equal(c, kept_c)
    assert not np.array_equal(held[-1][1], c)
    last = held[-1][1].copy()
    close()
    gc.collect()
    assert np.array_equal(held[-1][1], last) and np.array_equal(c, kept_c)
    c[:] = 0.0                      # writable, as a copy is
    assert np.array_equal(held[-1][1], last)
