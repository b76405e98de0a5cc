"""The EM-ICP pairs of a batch, each by a team of blocks of its own
(emicp_teams_kernel), against single calls: one pair over all blocks, teams of
many, odd and single blocks, several pairs on one block, more pairs than
blocks, sizes around the units of 128 and 512 points. The two cut the sums
differently; single calls are within 1e-3 degrees of the oracle and so is the
batch, hence 2e-3 between them, 1e-4 of the extent in translation."""
import numpy as np
import pytest

from conftest import rot_err_deg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [
    [(9001, 8003)],
    [(700, 127), (513, 129), (512, 128), (40, 33)],
    [(6007, 5003)] + [(1025, 640)] * 3 + [(300, 200 + k) for k in range(60)],
    [(257, 255)] * 400 + [(5001, 3001)],
])
def test_teams_agree_with_single_calls(cesa, sizes):
    from cuda_emicp_softassign_gb300 import workloads as W
    p = cesa.Params.default()
    pairs = []
    for k, (n, m) in enumerate(sizes):
        X, Y, _, _ = W.uniform_pair(n=n, m=m, seed=k % 5, max_deg=10.0, t_range=0.02)
        pairs.append((cesa.ALGO_EMICP, X, Y, p))
    single, res = {}, cesa.register_batch(pairs)
    for k, ((_, X, Y, _), (R, t)) in enumerate(zip(pairs, res)):
        key = (sizes[k], k % 5)
        if key not in single:
            single[key] = cesa.emicp(X, Y, param=p)
        assert rot_err_deg(R, single[key][0]) < 2e-3
        assert np.abs(t - single[key][1]).max() < 1e-4 * float(np.ptp(X, 0).max())


def test_pair_without_steps(cesa):
    """A pair whose schedule has no steps returns its initial pose; the others run."""
    from cuda_emicp_softassign_gb300 import workloads as W
    X, Y, _, _ = W.uniform_pair(n=600, m=500, seed=1, max_deg=10.0)
    none = cesa.Params.default(sigma_p2=1e-6, sigma_inf=1e-3)
    (R0, t0), (R1, t1) = cesa.register_batch([(cesa.ALGO_EMICP, X, Y, none),
                                              (cesa.ALGO_EMICP, X, Y, cesa.Params.default())])
    assert np.array_equal(R0, np.eye(3)) and np.array_equal(t0, np.zeros(3))
    Rs, ts = cesa.emicp(X, Y)
    assert rot_err_deg(R1, Rs) < 2e-3 and np.abs(t1 - ts).max() < 1e-4
