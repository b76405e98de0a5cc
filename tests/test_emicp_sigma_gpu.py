"""EM-ICP's E-step at the ends of sigma_p2's range, on column counts that end in part
groups: padding columns have no affinity, also where every real one's is 1. Rows
against the FP64 oracle, 1e-5."""
import numpy as np
import pytest
from conftest import rel_err, soa_tensor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sigma_p2", [1e-30, 1.0, 1e30, 1e34, 1e36, 3e38])
@pytest.mark.parametrize("n,m", [(1, 1), (100, 90), (513, 40), (9001, 50)])
def test_rows(cesa, oracle, torch_cuda, n, m, sigma_p2):
    from cuda_emicp_softassign_gb300 import workloads as W
    torch = torch_cuda
    X, Y, R, t = W.uniform_pair(n=n, m=m, seed=n)
    rows = torch.zeros(m * 5, dtype=torch.float32, device="cuda")
    cesa.emicp_step(soa_tensor(torch, X), soa_tensor(torch, Y), R, t, sigma_p2, 0.01, row_out=rows)
    got = rows.cpu().numpy().reshape(m, 5)
    ref = oracle.emicp_step(X, Y, R.astype(np.float32), t.astype(np.float32), float(np.float32(sigma_p2)), 0.01)
    assert rel_err(got[:, 0], ref["C"], floor=1e-30) < 1e-5
    assert rel_err(got[:, 1], ref["lam"]) < 1e-5
    assert rel_err(got[:, 2:], ref["U"]) < 1e-5
