"""The grid search's ball form (csrc/cesa_icp.cu) against the exhaustive search:
the same matches and, bitwise, the same pose, at sizes around its groups of 8
lanes, warps and shared sample of the target, for queries far outside the
grid (wide balls: a warp each), on flat and coincident targets and beside
points that are not finite (a query without a match takes the first point in
both)."""
import numpy as np
import pytest
from conftest import soa_tensor

pytestmark = pytest.mark.gpu


def _both(cesa, torch, X, Y, iters=6):
    out = []
    for search in (cesa.ICP_SEARCH_EXHAUSTIVE, cesa.ICP_SEARCH_GRID):
        p = cesa.Params.default(maxIteration=iters, icp_search=search)
        rt = torch.tensor([1, 0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0], dtype=torch.float32, device="cuda")
        nn = torch.full((len(Y),), -1, dtype=torch.int32, device="cuda")
        cesa.icp_device(soa_tensor(torch, X), soa_tensor(torch, Y), rt, p, d_nn=nn)
        torch.cuda.synchronize()
        out.append((rt.cpu().numpy(), nn.cpu().numpy()))
    return out


@pytest.mark.parametrize("n,m", [(1, 1), (2, 3), (65, 7), (1023, 9), (1025, 33), (5001, 2047), (300, 9001)])
@pytest.mark.parametrize("kind", ["surface", "far", "flat", "same"])
def test_equals_the_exhaustive_search(cesa, torch_cuda, n, m, kind):
    from cuda_emicp_softassign_gb300 import workloads as W
    X, Y, _, _ = W.surface_pair(n=n, m=m, seed=n + m, max_deg=20.0, outlier_frac=0.05)
    if kind == "far":
        Y[::3] += np.float32(1.0)
    elif kind == "flat":
        X[:, 2] = np.float32(0.25)
    elif kind == "same":
        X[:] = X[0]
    (a, na), (b, nb) = _both(cesa, torch_cuda, X, Y)
    assert np.array_equal(na, nb)
    if kind != "same" or n == 1:
        assert np.array_equal(a, b, equal_nan=True)
        return
    # a coincident target leaves the rotation free (the cross-covariance is
    # zero up to rounding): what is determined is that R is a rotation and
    # that Y's centroid lands on the point; |entries| <= 1, so a few FP32 ulp
    for rt in (a, b):
        R, t = rt[:9].reshape(3, 3).astype(np.float64), rt[9:].astype(np.float64)
        assert np.abs(R @ R.T - np.eye(3)).max() < 2e-6
        assert np.abs(R @ Y.astype(np.float64).mean(0) + t - X[0]).max() < 2e-6


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_points_that_are_not_finite(cesa, torch_cuda, value):
    from cuda_emicp_softassign_gb300 import workloads as W
    X, Y, _, _ = W.surface_pair(n=3000, m=1000, seed=5)
    Y[17, 1] = np.float32(value)
    if np.isnan(value):
        X[40, 2] = np.float32(value)
    (a, na), (b, nb) = _both(cesa, torch_cuda, X, Y, iters=1)
    assert np.array_equal(na, nb)
    assert np.array_equal(a, b, equal_nan=True)
