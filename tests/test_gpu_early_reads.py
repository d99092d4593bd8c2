"""The body kernel starts beside the contact pass and reads state of the step before (time, step, status,
displacement parameters, rigid bodies' state) ahead of its own wait.  Bodies of odd node counts, whose
arrays share memory sectors with their neighbours', stepped many times through proximity updates,
on as many bodies as there are SMs and a few more, so that bodies change SMs between steps: node state,
rigid state and works equal the oracle's bit for bit, alone and as a batch."""
import functools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@functools.lru_cache(maxsize=None)
def odd_flat():
    from melody2d_b200 import generator as g
    sc = g.disc_lattice_scene(seed=11, nx=13, ny=12, pitch=2.05e-3, gap0=-1e-6, n_border=24, n_interior=25,
                              min_sep=0.15e-3, v_plate=0.05)
    flat = g.flatten(sc)
    n = np.diff(flat["body_node_ptr"])[np.asarray(flat["body_type"]) == 0]
    assert len(n) == 156 and (n % 2 == 1).sum() >= 40
    return flat


@pytest.mark.parametrize("batch", [False, True])
def test_long_run_bit_identical(gpu_lib, oracle_built, batch):
    from melody2d_b200.solver import Batch, Solver
    from oracle.pyoracle import Oracle
    flat = odd_flat()
    s = Solver.from_flat(flat)
    o = Oracle(flat, correctly_rounded=True)
    b = None
    if batch:
        b = Batch(precision=0)
        b.admit(s)
    for _ in range(4):
        (b or s).step(75)
        o.step(75)
        np.testing.assert_array_equal(s.node_state(), o.node_state())
    np.testing.assert_array_equal(s.rigid()[0], o.rigid()[0])
    np.testing.assert_array_equal(s.works(), o.works())
    assert (s.contacts()["fx"] != 0).sum() > 20
    if b:
        b.close()
    s.close()
