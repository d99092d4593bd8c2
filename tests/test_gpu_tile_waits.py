"""The waits of the body kernel's pass over tiles, each made to run out by its own bound
(MELGPU_TILE_WAIT_NS, read when a model is created: the bound of the wait for a tile's index words and of
the one for its pull sections; -1 gives up without a look at the barrier, 0 looks once).  A wait that
gives up lets all warps of its CTA leave together: the step reports MEL_ERR_TIMEOUT, the context
stays usable and a fresh model steps as the oracle does.

With 0 for both waits it is up to the copies which threads find theirs in place, so that threads of one
CTA differ and the step may also come through."""
import numpy as np
import pytest

from conftest import flat_of, squeezed_lattice

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("bounds,certain", [("-1,999999999", True), ("999999999,-1", True), ("0,0", False)])
def test_tile_wait_gives_up(gpu_lib, oracle_built, monkeypatch, precision, bounds, certain):
    from melody2d_b200.solver import MelError, Solver
    from oracle.pyoracle import Oracle
    flat = flat_of(squeezed_lattice(3, 3))
    monkeypatch.setenv("MELGPU_TILE_WAIT_NS", bounds)
    s = Solver.from_flat(flat, precision=precision)
    code = 0
    try:
        s.step(1)
    except MelError as e:
        code = e.code
    assert code == 7 or (code == 0 and not certain)         # MEL_ERR_TIMEOUT
    assert (s.error_words()[6] != 0) == (code == 7)          # MEL_E_WAIT
    s.close()
    monkeypatch.delenv("MELGPU_TILE_WAIT_NS")
    g = Solver.from_flat(flat)
    o = Oracle(flat, correctly_rounded=True)
    g.step(20)
    o.step(20)
    np.testing.assert_array_equal(g.node_state(), o.node_state())
    g.close()
