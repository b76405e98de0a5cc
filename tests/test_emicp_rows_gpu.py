"""EM-ICP on small clouds (emicp_rows_kernel: whole rows to a block, X in shared
memory) against the FP64 oracle, at sizes around its passes of 4 rows, its
blocks of 4, 8 and up to 32, its columns padded to 512 and the most that it
takes (8192), and against a batch of one pair (which takes the other forms).

Tolerance: a final rotation within 1e-3 degrees of the oracle and translation
within 1e-5 of the extent (as the other forms), so 2e-3 and 2e-5 between two
forms; twice the reference's own FP32 arithmetic where a pair is
ill-conditioned."""
import numpy as np
import pytest

from conftest import rot_err_deg

pytestmark = pytest.mark.gpu


def _pair(n, m, seed):
    from cuda_emicp_softassign_gb300 import workloads as W
    X, Y, _, _ = W.uniform_pair(n=n, m=m, seed=seed, max_deg=10.0, t_range=0.02)
    return X, Y


@pytest.mark.parametrize("n,m", [(33, 5), (600, 8), (512, 129), (513, 609), (1023, 1217), (300, 3000), (8192, 41)])
def test_sizes(cesa, oracle, n, m):
    X, Y = _pair(n, m, n + m)
    R, t = cesa.emicp(X, Y)
    Ro, to, _ = oracle.emicp(X, Y, trace=False)
    Rp, tp, _ = oracle.emicp(X, Y, precision="f32", trace=False)
    assert rot_err_deg(R, Ro) <= max(1e-3, 2 * rot_err_deg(Rp, Ro))
    assert np.abs(t - to).max() <= max(1e-5 * float(np.ptp(X, 0).max()), 2 * np.abs(tp - to).max())


@pytest.mark.parametrize("n,m", [(700, 2433), (8192, 1216), (4001, 4001), (8191, 8500), (8193, 600), (7000, 10100)])
def test_agrees_with_the_other_forms(cesa, n, m):
    X, Y = _pair(n, m, 3)
    R, t = cesa.emicp(X, Y)
    (Rb, tb), = cesa.register_batch([(cesa.ALGO_EMICP, X, Y, cesa.Params.default())])
    assert rot_err_deg(R, Rb) < 2e-3
    assert np.abs(t - tb).max() < 2e-5 * float(np.ptp(X, 0).max())


@pytest.mark.parametrize("cloud", [0, 1])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_points_that_are_not_finite(cesa, cloud, value):
    """They reach the pose, or do not, as in the other forms."""
    clouds = [c.copy() for c in _pair(600, 500, 4)]
    clouds[cloud][7, 1] = value
    R, t = cesa.emicp(*clouds)
    (Rb, tb), = cesa.register_batch([(cesa.ALGO_EMICP, *clouds, cesa.Params.default())])
    assert np.isfinite(R).all() == np.isfinite(Rb).all() and np.isfinite(t).all() == np.isfinite(tb).all()
