"""The order of a batch's body CTAs (most work first over all members, in the launch of the members that
fit two CTAs per SM and in the launch of the others): a member's state is the one it has alone, with
members on both sides of that line, of uneven bodies, alone in their class or not."""
import numpy as np
import pytest

from conftest import flat_of, squeezed_lattice
from test_gpu_batch import assert_same, state

pytestmark = pytest.mark.gpu


def _members(which):
    from melody2d_b200 import generator as g
    draws = dict(grains=(10, 10), border=(32, 60))
    counts = g.batch_sample_params(7, **draws)["n_border"]
    make = {"lattice": lambda: flat_of(squeezed_lattice(3, 3)),
            "uneven": lambda: g.flatten(g.batch_sample_scene(7, g.DiscTemplates(counts, workers=1), **draws)),
            "large": lambda: g.flatten(g.biaxial_scene(seed=8, n_discs=3, n_border=96, n_interior=900, workers=1))}
    return [make[w]() for w in which]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("which", [("large",), ("large", "uneven"), ("lattice", "large", "uneven", "large")])
def test_members_equal_alone(gpu_lib, which, precision):
    from melody2d_b200.solver import Batch, Solver
    flats = _members(which)
    b = Batch(precision=precision)
    mixed = [Solver.from_flat(f, precision=precision) for f in flats]
    for s in mixed:
        b.admit(s)
    b.step(12)
    b.retire(mixed[0])
    b.step(5)
    for k, (f, t) in enumerate(zip(flats, mixed)):
        s = Solver.from_flat(f, precision=precision)
        s.step(12 if k == 0 else 17)
        assert_same(state(s), state(t))
    b.close()
