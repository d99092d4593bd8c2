"""Row pointers of the shape functions where the scan of the support counts takes one stride of 8,192 counts
or several: they equal the sums of the counts found by numpy.  (The scan's indices are 64 bits wide, as
they have to be for point counts within a stride of the largest int; such a call is too large for a test.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points", [(8191,), (8192,), (8193,), (16383, 2), (5000, 0, 20001)])
def test_row_pointers(gpu_lib, points):
    from melody2d_b200.solver import mls_shapes
    rng = np.random.default_rng(sum(points))
    g = (np.arange(5) - 2.0) / 5
    nodes = np.stack(np.meshgrid(g, g), -1).reshape(-1, 2)
    jobs = [(rng.uniform(-0.4, 0.4, (n, 2)), nodes, rng.uniform(0.5, 0.6, 25)) for n in points]
    for (pts, x, r), d in zip(jobs, mls_shapes(jobs)):
        rel = pts[:, None, :] - x[None, :, :]
        inside = (rel[..., 0] * rel[..., 0] + rel[..., 1] * rel[..., 1]) - r[None, :] * r[None, :] < 0.0
        np.testing.assert_array_equal(d[0], np.concatenate([[0], np.cumsum(inside.sum(axis=1))]))
        np.testing.assert_array_equal(d[1], np.nonzero(inside)[1])
