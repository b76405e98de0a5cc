"""The ICP grid search on targets of uneven extents (csrc/cesa_icp.cu): tubes,
corridors and lines along every axis, and very large coordinates. The grid has to
cover its target and a search to reach every cell that can hold a match: matches
and (bitwise) poses are the exhaustive search's, in the first iteration, which
starts from a sample of the target, and in later ones, which start from the
previous match."""
import numpy as np
import pytest
from test_icp_ball_gpu import _both

pytestmark = pytest.mark.gpu


def _box(n, m, extents, seed):
    """Points uniform in a box; every seventh query beyond its ends."""
    rng = np.random.default_rng(seed)
    e = np.asarray(extents, np.float64)
    X, Y = rng.uniform(0, 1, (n, 3)) * e, rng.uniform(0, 1, (m, 3)) * e
    Y[::7] = Y[::7] * 1.5 - 0.25 * e
    return X.astype(np.float32), Y.astype(np.float32)


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n,m,extents", [
    (5000, 9000, (1, 0.001, 0.001)),   # the automatic choice takes the grid from here on
    (40000, 4000, (1, 0.001, 0.001)),
    (40097, 4000, (1, 0.005, 0.005)),
    (40097, 4000, (100, 0.5, 0.5)),
    (200000, 2000, (1, 0.015, 0.015)),
    (250000, 1000, (100, 2, 2)),       # a corridor
    (40000, 4000, (1, 1, 0.3)),
    (64, 300, (1, 0.001, 0.001)),      # the fewest cells
])
def test_equals_the_exhaustive_search(cesa, torch_cuda, n, m, extents, axis):
    X, Y = _box(n, m, np.roll(extents, axis), seed=n + axis)
    for iters in (1, 5):
        (a, na), (b, nb) = _both(cesa, torch_cuda, X, Y, iters=iters)
        assert np.array_equal(na, nb)
        assert np.array_equal(a, b)


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n", [10000, 40000])
def test_collinear_target(cesa, torch_cuda, n, axis):
    """(a line leaves the rotation about it free: one iteration's matches)"""
    X, Y = _box(n, 4000, np.roll((1, 0, 0), axis), seed=n + axis)
    Y += np.float32(0.01)
    (_, na), (_, nb) = _both(cesa, torch_cuda, X, Y, iters=1)
    assert np.array_equal(na, nb)


@pytest.mark.parametrize("scale", [1e-12, 1e15, 1e17, 1e19])
def test_scales(cesa, torch_cuda, scale):
    """Squared distances of 1e30 and above count like any other; at 1e19 most
    overflow (a query whose distances are all infinite takes the first point)."""
    X, Y = _box(40000, 2000, (1, 1, 0.3), seed=9)
    (_, na), (_, nb) = _both(cesa, torch_cuda, X * np.float32(scale), Y * np.float32(scale), iters=1)
    assert np.array_equal(na, nb)
