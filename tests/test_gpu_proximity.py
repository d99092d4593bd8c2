"""Update_proximity where its launches change form: one member's job as the kernels' argument, a table
of a few members, and more members than a scan takes as its argument; and a candidate list that
outgrows its first allocation (some 2,200 candidates).  Contact lists equal those of the same samples
alone, and the oracle's."""
import numpy as np
import pytest

from conftest import flat_of
from test_gpu_parity import assert_contacts_equal

pytestmark = pytest.mark.gpu


def lattice(seed, nx=2, ny=1):
    from melody2d_b200 import generator as g
    return g.disc_lattice_scene(seed=seed, nx=nx, ny=ny, pitch=2.05e-3, gap0=-1e-6, n_border=24, n_interior=24, min_sep=0.15e-3)


@pytest.mark.parametrize("members", [1, 2, 6])
def test_members_of_one_run(gpu_lib, oracle_built, members):
    from melody2d_b200 import generator as g
    from melody2d_b200.solver import Batch, Solver
    from oracle.pyoracle import Oracle
    flats = [g.flatten(lattice(seed, nx=2 + seed % 3)) for seed in range(members)]
    solvers = [Solver.from_flat(f) for f in flats]
    b = Batch()
    for s in solvers:
        b.admit(s)
    assert b.step(25) == []
    for s, f in zip(solvers, flats):
        o = Oracle(f, correctly_rounded=True)
        o.step(25)
        assert_contacts_equal(s.contacts(), o.contacts())
        np.testing.assert_array_equal(s.node_state(), o.node_state())
    b.close()
    for s in solvers:
        s.close()


def test_candidate_list_grows(gpu_lib, oracle_built):
    from melody2d_b200 import generator as g
    from melody2d_b200.solver import Solver
    from oracle.pyoracle import Oracle
    sc = g.disc_lattice_scene(seed=0, nx=8, ny=8, pitch=2.05e-3, gap0=-1e-6, n_border=48, n_interior=40, min_sep=0.1e-3)
    for body in sc.bodies:
        body.detection = body.contact = 9.0 * body.detection      # many nodes near the next disc
    flat = g.flatten(sc)
    o = Oracle(flat, correctly_rounded=True)
    assert len(o.contacts()) > 2500
    s = Solver.from_flat(flat)
    assert_contacts_equal(s.contacts(), o.contacts())
    s.step(11)
    o.step(11)
    assert_contacts_equal(s.contacts(), o.contacts())
    s.close()
