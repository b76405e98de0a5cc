"""EM-ICP's local sweep (csrc/cesa_emicp.cu: Y sorted along a Hilbert curve,
blocks of 128 rows about their own centres), which clouds from 2.4e7
affinities a step on take: one E-step against the FP64 oracle, per row in the
caller's order and in its moments. The sizes end in part blocks and part
chunks; 20,001 x 16,300 is swept in ranges. sigma_p2 from 1e-2 (every block in
the short form) to 1e-5 (most blocks by direct differences), on surfaces and on
a unit cube. Tolerances as for the plain sweep (test_emicp_gpu.py): per row
1e-5 or twice the error of the reference's FP32 arithmetic, moments 1e-5."""
import numpy as np
import pytest
from conftest import rel_err, soa_tensor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sigma_p2", [1e-2, 3e-4, 1.06e-5])
@pytest.mark.parametrize("n,m,gen", [(6000, 4097, "surface"), (4700, 5200, "cube"), (129, 190001, "surface"),
                                     (20001, 16300, "surface")])
def test_estep_rows_and_moments(cesa, oracle, torch_cuda, n, m, gen, sigma_p2):
    from cuda_emicp_softassign_gb300 import workloads as W
    torch = torch_cuda
    if gen == "cube":
        X, Y, R, t = W.uniform_pair(n=n, m=m, seed=n + m)
    else:
        X, Y, R, t = W.surface_pair(n=n, m=m, seed=n + m, max_deg=20.0, outlier_frac=0.05)
    assert float(n) * m >= 2.4e7
    dX, dY = soa_tensor(torch, X), soa_tensor(torch, Y)
    rows = torch.zeros(m * 5, dtype=torch.float32, device="cuda")
    mom = cesa.emicp_step(dX, dY, R, t, sigma_p2, 0.01, row_out=rows)
    got = rows.cpu().numpy().reshape(m, 5)
    ref = oracle.emicp_step(X, Y, R.astype(np.float32), t.astype(np.float32), sigma_p2, 0.01)
    port = oracle.emicp_step(X, Y, R.astype(np.float32), t.astype(np.float32), sigma_p2, 0.01, precision="f32")

    def worst(a, b, floor):
        return float((np.abs(a - b) / np.maximum(np.abs(b), floor)).max())

    for col, key, floor in ((0, "C", 1e-30), (1, "lam", 1e-3)):
        e_gpu, e_port = worst(got[:, col], ref[key], floor), worst(port[key], ref[key], floor)
        assert e_gpu <= max(1e-5, 2.0 * e_port), (key, e_gpu, e_port)
    e_gpu, e_port = rel_err(got[:, 2:5], ref["U"]), rel_err(port["U"], ref["U"])
    assert e_gpu <= max(1e-5, 2.0 * e_port), ("U", e_gpu, e_port)
    extent = float(np.ptp(X, 0).max())
    assert abs(mom[0] - ref["sum"]) <= 1e-5 * ref["sum"]
    assert np.abs(mom[1:4] - ref["Xc"]).max() < 1e-5 * extent
    assert np.abs(mom[4:7] - ref["Yc"]).max() < 1e-5 * extent
    assert rel_err(mom[7:16], ref["S"]) < 1e-5


@pytest.mark.parametrize("case", ["same", "line", "nan", "inf"])
def test_degenerate_clouds_as_the_plain_sweep(cesa, case):
    """Coincident and collinear points sort and sweep; a coordinate that is not
    finite gives a pose that is not finite in the same places as just below
    the local sweep's sizes."""
    def run(n):
        rng = np.random.default_rng(3)
        X = rng.uniform(0, 0.2, (n, 3)).astype(np.float32)
        Y = X.copy()
        if case == "same":
            Y[:] = Y[0]
        elif case == "line":
            Y[:, 1:] = 0.1
        else:
            Y[7, 2] = np.float32(case)
        return cesa.emicp(X, Y, param=cesa.Params.default(sigma_inf=5e-3))
    (R1, t1), (R2, t2) = run(5000), run(4800)
    assert np.array_equal(np.isfinite(R1), np.isfinite(R2)) and np.array_equal(np.isfinite(t1), np.isfinite(t2))
