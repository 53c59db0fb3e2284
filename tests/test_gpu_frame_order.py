"""A frame formed at once (sww_frame) in between leaves the asynchronous frame
that was started last as it was: waiting for it again gives the same values,
whether its buffer was handed over or not (exact comparisons)."""
import numpy as np
import pytest

from anuga_core_gb300.workloads import dam_break

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first_wait", [True, False])
@pytest.mark.parametrize("m", [1, 24])
def test_immediate_frame_between_waits(m, first_wait):
    d = dam_break(m, "DE1", precision="fp64")
    flat = d.mesh.triangles.ravel()
    off = np.zeros(d.mesh.number_of_nodes + 1, np.int64)
    off[1:] = np.cumsum(np.bincount(flat, minlength=d.mesh.number_of_nodes))
    d.advance_steps(1)
    scn = d._scn
    scn.sww_bind(off, np.argsort(flat, kind="stable"))
    v0, c0 = scn.sww_frame(1.0e-3)
    scn.sww_frame_async(1.0e-3)
    if first_wait:
        v, c = scn.sww_frame_wait()
        assert np.array_equal(v, v0) and np.array_equal(c, c0)
    d.advance_steps(3)
    v1, c1 = scn.sww_frame(1.0e-3)
    assert not np.array_equal(c1, c0)
    v, c = scn.sww_frame_wait()
    assert np.array_equal(v, v0) and np.array_equal(c, c0)
    scn.sww_frame_async(1.0e-3)
    v, c = scn.sww_frame_wait()
    assert np.array_equal(v, v1) and np.array_equal(c, c1)
