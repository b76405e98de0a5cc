"""How far emicp_step's row sums are from FP64 (csrc/cesa_emicp.cu): no further than
those of direct differences in FP32 (each posed point rounded per operation, a
difference, its square and the exponent's scale rounded once each, the exponential
and the sums exact, so for up to some 10,000 columns, whose FP32 sums add little). That
arithmetic is emulated here, over the same rows."""
import numpy as np
import pytest
from conftest import soa_tensor

pytestmark = pytest.mark.gpu
F = np.float32


def _direct(X, Y, R, t, s2):
    """Row sums of e^2 by direct differences: in FP64, and in emulated FP32 about the clouds' means."""
    oX, oY = X.mean(0).astype(F), Y.mean(0).astype(F)
    x, y = (X - oX).astype(F), (Y - oY).astype(F)
    R64, s = R.astype(np.float64), float(F(s2))
    tc = (R64 @ oY.astype(np.float64) + t - oX).astype(F)
    z = np.empty_like(y)
    for i in range(3):
        a = (R[i, 0] * y[:, 0]).astype(F)
        for j in (1, 2):
            a = (float(R[i, j]) * y[:, j].astype(np.float64) + a).astype(F)
        z[:, i] = (a + tc[i]).astype(F)
    exact = np.zeros(len(Y))
    z64 = Y.astype(np.float64) @ R64.T + t
    emul = np.zeros(len(Y))
    nk = F(-np.log2(np.e) / (2 * s))
    for k in range(len(Y)):
        exact[k] = np.exp(-((X.astype(np.float64) - z64[k]) ** 2).sum(1) / s).sum()
        d = (x - z[k]).astype(F)
        q = (d[:, 0] * d[:, 0]).astype(F)
        for j in (1, 2):
            q = (d[:, j].astype(np.float64) ** 2 + q).astype(F)
        emul[k] = np.exp2(2.0 * (nk * q).astype(F).astype(np.float64)).sum()
    out = np.exp(-0.01 / s)
    return exact + out, emul + out


@pytest.mark.parametrize("sigma_p2", [1e-4, 1.06e-5])
@pytest.mark.parametrize("n,m", [(2000, 2000), (8171, 6007), (10007, 9001)])
def test_rows_are_as_near_as_direct_differences(cesa, torch_cuda, n, m, sigma_p2):
    from cuda_emicp_softassign_gb300 import workloads as W
    torch = torch_cuda
    e_gpu = e_emul = 0.0
    for seed in (1, 2, 3):
        X, Y, R, t = W.surface_pair(n=n, m=m, seed=seed, max_deg=20.0, outlier_frac=0.05)
        R, t = R.astype(F), t.astype(F)
        rows = torch.zeros(m * 5, dtype=torch.float32, device="cuda")
        cesa.emicp_step(soa_tensor(torch, X), soa_tensor(torch, Y), R, t, sigma_p2, 0.01, row_out=rows)
        pick = np.random.default_rng(seed).permutation(m)[:600]
        got = rows.cpu().numpy().reshape(m, 5)[pick, 0].astype(np.float64)
        exact, emul = _direct(X, Y[pick], R, t.astype(np.float64), sigma_p2)
        scale = np.maximum(exact, 1e-3)
        e_gpu += (((got - exact) / scale) ** 2).mean()
        e_emul += (((emul - exact) / scale) ** 2).mean()
    # 10%: the spread of a mean over 1800 rows
    assert np.sqrt(e_gpu) <= 1.1 * np.sqrt(e_emul), (np.sqrt(e_gpu / 3), np.sqrt(e_emul / 3))
