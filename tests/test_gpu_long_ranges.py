"""Rigid bodies whose contacts come in long lists: a block sheared along another has all its incoming contacts
in one range.  Range lengths on both sides of what one thread copies alone (8), of what the kernel stages
at once (1,024) and of the threads' count (256 ranges), against the oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def blocks_flat(n, discs=0):
    """Two rigid blocks face to face, n border nodes along the shared side, the upper one pressed on the
    lower and sheared along it; a small deformable disc apart; `discs` rigid ones in a row on the upper block."""
    import random
    from melody2d_b200 import generator as g
    L = 0.1
    h = L / n
    hist = lambda v: (np.array([0.0, g.T_HIST_END]), np.array([v, v]))
    bc = lambda v: (g.BC_DRIVEN, (0.0, 0.0), hist(v))
    mats = [("Steel", 0, [7800.0, 0.0, 0.0, 2e11, 0.3, 500.0])]
    laws = [("Steel", "Steel", 2, 0, [1e10, 1e9, 0.3, 0.0, 0.0])]
    a = g.make_rect_rigid(0, -0.01, L, 0.0, h, 0, 7800.0, bc(0.0), bc(0.0), 0.7 * h, 0.7 * h)
    b = g.make_rect_rigid(0.13 * h, -0.01 * h, L + 0.13 * h, 0.01, h, 0, 7800.0, bc(0.01), bc(-0.001), 0.7 * h, 0.7 * h)
    bodies = [g.make_disc(random.Random(1), (0.05, 0.05), 1e-3, 24, 40, 0.15e-3, 0, 2500.0), a, b]
    for k in range(discs):
        r = 0.4 * L / discs
        bodies.append(g.make_rigid_disc(((k + 0.5) * L / discs, 0.01 + 0.99 * r), r, 12, 0, 7800.0, 0.3 * r, 0.3 * r))
    return g.flatten(g.Scene(name="blocks", bodies=bodies, materials=mats, laws=laws, dt=1e-9, nsteps=100,
                             contact_update_period=1e-8))


def longest(c, body):
    """Lengths of the runs of contacts with one slave body and master `body`."""
    s = c["bodyS"][c["bodyM"] == body]
    return np.bincount(s).max() if len(s) else 0


@pytest.mark.parametrize("n,discs,at_least", [(6, 0, 6), (8, 0, 8), (9, 0, 9), (300, 0, 300), (1022, 0, 1022), (1024, 0, 1024),
                                              (1026, 0, 1025), (2100, 0, 2049), (12, 300, 9), (700, 300, 700)])
def test_long_incoming_ranges(gpu_lib, oracle_built, n, discs, at_least):
    from melody2d_b200.solver import Solver
    from oracle.pyoracle import Oracle
    from test_gpu_parity import assert_contacts_equal
    flat = blocks_flat(n, discs)
    s = Solver.from_flat(flat)
    o = Oracle(flat, correctly_rounded=True)
    for _ in range(2):
        s.step(12)
        o.step(12)
        assert_contacts_equal(s.contacts(), o.contacts())
        np.testing.assert_array_equal(s.rigid()[0], o.rigid()[0])
        np.testing.assert_array_equal(s.rigid()[1], o.rigid()[1])
        np.testing.assert_array_equal(s.node_state(), o.node_state())
    c = s.contacts()
    assert longest(c, 1) >= at_least and (c["fx"] != 0).sum() > 4
    if discs:
        assert len(np.unique(c["bodyS"][c["bodyM"] == 2])) > 256
    np.testing.assert_array_equal(s.works(), o.works())
    s.close()
