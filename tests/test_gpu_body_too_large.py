"""Bodies a little above the largest that test_gpu_body_limits takes, whose node arrays would fit a CTA alone but
not beside the descriptor that a batch's CTAs hold: refused as other bodies without room are, not by a
failing CUDA call, and models of the same process step afterwards."""
import numpy as np
import pytest

from conftest import flat_of, squeezed_lattice

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,nodes", [(0, 1314), (0, 1319), (0, 1330), (1, 1257), (1, 1262), (1, 1270)])
def test_refused_as_unsupported(gpu_lib, oracle_built, precision, nodes):
    from melody2d_b200 import generator as g
    from melody2d_b200.solver import MelError, Solver
    from oracle.pyoracle import Oracle
    flat = g.flatten(g.biaxial_scene(seed=9, n_discs=2, n_border=100, n_interior=nodes - 100, workers=1))
    assert np.diff(flat["body_node_ptr"]).max() == nodes
    with pytest.raises(MelError) as e:
        Solver.from_flat(flat, precision=precision)
    assert e.value.code == 2 and "%d nodes does not fit" % nodes in str(e.value)        # MEL_ERR_UNSUPPORTED
    small = flat_of(squeezed_lattice(2, 2))
    s = Solver.from_flat(small)
    o = Oracle(small, correctly_rounded=True)
    s.step(10)
    o.step(10)
    np.testing.assert_array_equal(s.node_state(), o.node_state())
    s.close()
