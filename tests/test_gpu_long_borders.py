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


@pytest.mark.parametrize("n", [40, 126, 127, 128, 252, 254, 256, 900])
def test_history_of_long_lists(gpu_lib, oracle_built, n):
    """Lists handed in by the caller, each contact twice with different history and in any order within its
    slave body: on both sides of 256 elements a body, an update inherits from the first in the list."""
    from melody2d_b200.solver import Solver
    from oracle.pyoracle import Oracle
    flat = blocks_flat(n)
    s = Solver.from_flat(flat)
    o = Oracle(flat, correctly_rounded=True)
    c = s.contacts()
    rng = np.random.default_rng(n)
    twice = np.concatenate([c, c])
    twice["gapt"] = rng.standard_normal(len(twice))
    twice["vgapt"] = rng.standard_normal(len(twice))
    twice = twice[np.lexsort((rng.random(len(twice)), twice["bodyS"]))]
    for x in (s, o):
        x.set_contacts(twice)
        x.update_proximity()
    assert_contacts_equal(s.contacts(), o.contacts())
    assert len(np.unique(s.contacts()["gapt"])) > n // 2
    # and from the list that this left
    for x in (s, o):
        x.step(11)
    assert_contacts_equal(s.contacts(), o.contacts())
    s.close()
