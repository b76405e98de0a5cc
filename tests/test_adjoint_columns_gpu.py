"""The EM-ICP backward with 2 columns a lane (small clouds) against the 6 of the
forced ranged layout, over the same forward, at sizes around its units of 512
columns and 64 rows. Both are FP32 with errors of some 1e-5 of the largest
gradient against FP64 (66 steps), so 1e-4 between them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(40, 33), (511, 65), (513, 128), (1007, 1007), (1536, 2049), (4001, 3999)])
def test_two_columns_a_lane(cesa, torch_cuda, n, m):
    from cuda_emicp_softassign_gb300 import workloads as W
    from cuda_emicp_softassign_gb300.autograd import emicp_autograd
    torch = torch_cuda
    X, Y, Rt, _ = W.uniform_pair(n=n, m=m, seed=n, max_deg=10.0, t_range=0.02)
    grads = []
    for layout in (cesa.LAYOUT_AUTO, cesa.LAYOUT_RANGED):
        leaves = [torch.tensor(v, dtype=torch.float32, device="cuda", requires_grad=True)
                  for v in (X, Y, np.eye(3), np.zeros(3))]
        R, t = emicp_autograd(*leaves, cesa.Params.default(emicp_backward_layout=layout))
        (((R - torch.tensor(Rt, dtype=torch.float32, device="cuda")) ** 2).sum() + (t ** 2).sum()).backward()
        grads.append([v.grad.cpu().numpy() for v in leaves])
    # where the registration has converged the initial pose's gradient vanishes
    # (1e-41): it counts against the size of the clouds' gradients
    floor = np.abs(grads[1][0]).max()
    for k, (a, b) in enumerate(zip(*grads)):
        assert np.isfinite(a).all()
        assert np.abs(a - b).max() <= 1e-4 * max(np.abs(b).max(), floor if k >= 2 else 0.0)
