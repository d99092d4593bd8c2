"""Shape functions on the device where a body's points split over thread blocks (128 a block) and a point's
supports over a warp's lanes (32): point counts on both sides of a block's share, supports from a few to all
of a body's nodes, one body or several in a call, against the host's pass."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# host and device solve the same 3x3 systems in other bases; nodes about the origin with radii of the
# body's own size keep the host's basis conditioned to ~1e-3 at worst, so 1e-9 of the largest value bounds
# both roundings
TOL = 1e-9


def _job(rng, n_points, side, reach):
    g = (np.arange(side) - 0.5 * (side - 1)) / side
    nodes = np.stack(np.meshgrid(g, g), -1).reshape(-1, 2) + rng.uniform(-0.15, 0.15, (side * side, 2)) / side
    radii = rng.uniform(0.9, 1.1, side * side) * reach / side
    return rng.uniform(-0.45, 0.45, (n_points, 2)), nodes, radii


@pytest.mark.parametrize("points", [(1,), (127,), (128,), (129,), (0, 1, 257, 0, 128, 31)])
@pytest.mark.parametrize("side,reach", [(5, 2.5), (12, 3.4), (12, 3.9), (9, 20.0)])
def test_slices_and_long_supports(gpu_lib, monkeypatch, points, side, reach):
    from melody2d_b200 import generator
    from melody2d_b200.solver import mls_shapes
    # the host looks among a point's 40 nearest nodes, which can miss a support with a larger radius: all here
    monkeypatch.setattr(generator._supports, "__defaults__", (10**6,))
    rng = np.random.default_rng(1000 * len(points) + 10 * points[-1] + side)
    jobs = [_job(rng, n, side, reach) for n in points]
    for (pts, nodes, radii), d in zip(jobs, mls_shapes(jobs)):
        assert len(d[0]) == len(pts) + 1
        if not len(pts):
            assert len(d[1]) == 0
            continue
        h = generator.mls_shape(pts, nodes, radii, np.zeros(2))
        np.testing.assert_array_equal(d[0], h[0])
        np.testing.assert_array_equal(d[1], h[1])
        for a, b in zip(d[2:], h[2:]):
            assert np.abs(a - b).max() <= TOL * np.abs(b).max()
