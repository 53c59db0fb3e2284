"""Plain FP64 step kernels at the sizes where their blocks end and their
dispatch changes: meshes of 4 to a few hundred triangles around the kernels'
32- and 128-cell blocks, and of 19,800 and 20,200, three steps of each flow algorithm without friction, bit for bit the
oracle's (no tolerance: the FP64 form rounds every operation as the oracle
does)."""
import numpy as np
import pytest

from anuga_core_gb300.mesh import Mesh, rectangular_cross
from helpers import make_domain, make_oracle, random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alg", ["DE0", "DE1", "DE2", "DE0_7"])
# the last two sit on both sides of the 20,000 cells from which the kernels form products with integer instructions
@pytest.mark.parametrize("m,n", [(1, 1), (7, 1), (8, 1), (9, 1), (4, 4), (17, 1), (8, 4), (3, 11), (16, 16), (13, 21),
                                 (99, 50), (101, 50)])
def test_steps_bitwise_at_block_ends(oracle_mod, alg, m, n):
    p, e, b = rectangular_cross(m, n, 10.0 * m, 10.0 * n)
    mesh = Mesh(p, e, b)
    st = random_state(mesh, 7 * m + n)
    st["friction"][:] = 0.0
    kinds = {"left": ("dirichlet", (1.0, 0.1, 0.0)), "right": ("transmissive", None),
             "top": ("reflective", None), "bottom": ("reflective", None)}
    d = make_domain(p, e, b, alg, st, kinds)
    od = make_oracle(oracle_mod, mesh, alg, st, kinds)
    for _ in od.evolve(yieldstep=1.0e9, finaltime=2.0e9, max_steps=3):
        pass
    d.distribute_to_vertices_and_edges()
    d.update_boundary()
    d.advance_steps(3)
    d.distribute_to_vertices_and_edges()
    assert d.total_steps == od.total_steps == 3
    for name, ref in (("stage", od.stage_c), ("xmomentum", od.xmom_c), ("ymomentum", od.ymom_c)):
        got = d.quantities[name].centroid_values
        assert np.array_equal(got, ref), name
