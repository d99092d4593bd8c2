"""Contact detection along long borders: two blocks face to face whose borders have one superblock of
segment boxes (256 segments), a few, and more than the 32 that a warp tests at a time.  The contact lists of
the set-up and of updates after it equal the oracle's, element by element, history included."""
import numpy as np
import pytest

from test_gpu_long_ranges import blocks_flat
from test_gpu_parity import assert_contacts_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,superblocks", [(110, 1), (120, 2), (700, 7), (3700, 32), (4300, 37)])
def test_contact_lists(gpu_lib, oracle_built, n, superblocks):
    from melody2d_b200.solver import Solver
    from oracle.pyoracle import Oracle
    flat = blocks_flat(n)
    assert (np.diff(flat["border_node_ptr"])[1] - 1 + 255) // 256 == superblocks
    s = Solver.from_flat(flat)
    o = Oracle(flat, correctly_rounded=True)
    assert_contacts_equal(s.contacts(), o.contacts())
    s.step(11)
    o.step(11)
    assert_contacts_equal(s.contacts(), o.contacts())
    assert (s.contacts()["fx"] != 0).sum() > n
    s.close()
