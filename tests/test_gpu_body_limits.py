"""The largest bodies whose node arrays fit the body kernel's shared memory, alone and in a batch (whose CTAs
also hold the member's descriptor): they are taken, and step as the oracle does (FP64 bit for bit, the
mixed form within its own bound)."""
import numpy as np
import pytest

from test_gpu_large_body import seeded_state

pytestmark = pytest.mark.gpu

TOL_MIXED = 1e-5         # the mixed form's stated tolerance


@pytest.mark.parametrize("precision,nodes,batch", [(0, 1313, False), (0, 1313, True), (1, 1256, False), (1, 1256, True)])
def test_largest_bodies_step(gpu_lib, oracle_built, precision, nodes, batch):
    from melody2d_b200 import generator as g
    from melody2d_b200.solver import Batch, Solver
    from oracle.pyoracle import Oracle
    flat = g.flatten(g.biaxial_scene(seed=9, n_discs=2, n_border=100, n_interior=nodes - 100, workers=1))
    assert np.diff(flat["body_node_ptr"]).max() == nodes
    o = Oracle(flat, correctly_rounded=True)
    s = Solver.from_flat(flat, precision=precision)
    st = seeded_state(flat, o.node_state())
    s.set_node_state(st)
    o.set_node_state(st)
    if batch:
        b = Batch(precision=precision)
        b.admit(s)
        b.step(12)
    else:
        s.step(12)
    o.step(12)
    got, want = s.node_state(), o.node_state()
    if precision == 0:
        np.testing.assert_array_equal(got, want)
    else:
        for cols in (slice(0, 2), slice(2, 4)):             # displacements, velocities
            assert np.abs(got[:, cols] - want[:, cols]).max() <= TOL_MIXED * np.abs(want[:, cols]).max()
    if batch:
        b.close()
