"""Which form an EM-ICP registration takes (csrc/cesa_emicp.cu) and, at sizes that do
take it, the local form: its E-step from any pose against the FP64 oracle (the first
record of a registration's trace; the sizes end in part blocks and part chunks, two
are swept in ranges), its gradients in the caller's row order, and coordinates that
coincide or are not finite. Moments' tolerances as for the single E-step
(test_emicp_local_gpu.py): 1e-5."""
import numpy as np
import pytest
from conftest import rel_err, soa_tensor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,sigma_inf,form", [
    (100, 100, 1e-5, "ROWS"), (1007, 1007, 1e-5, "ROWS"), (8171, 6007, 1e-5, "ROWS"),
    (9001, 9001, 1e-5, "LOCAL"), (8193, 6390, 1e-5, "LOCAL"), (40097, 40097, 1e-5, "LOCAL"),
    (3000, 100000, 1e-5, "LOCAL"), (100000, 9000, 1e-5, "LOCAL"),
    # many rows to a block against few columns: the second barrier costs less
    (16, 7000, 1e-5, "SLICES"), (100, 9000, 1e-5, "SLICES"), (600, 9000, 1e-5, "SLICES"), (16, 5000, 1e-5, "ROWS"),
    (300, 9700, 1e-5, "ROWS"), (1000, 8000, 1e-5, "ROWS"), (2000, 9700, 1e-5, "ROWS"),
    # few affinities a step: the refined poses and the sort cost more than the shorter element saves
    (9000, 2700, 1e-5, "SLICES"), (190001, 129, 1e-5, "SLICES"),
    # few columns to a row, or few steps: the sort costs more
    (129, 190001, 1e-5, "SLICES"), (1000, 50000, 1e-5, "SLICES"), (1000, 400000, 1e-5, "RANGES"),
    (30, 1000000, 1e-5, "RANGES"), (40097, 40097, 0.0095, "RANGES"), (10007, 9001, 0.0095, "SLICES"),
])
def test_form_by_size(cesa, torch_cuda, n, m, sigma_inf, form):
    assert cesa.emicp_form(n, m, cesa.Params.default(sigma_inf=sigma_inf)) == getattr(cesa, "EMICP_FORM_" + form)


@pytest.mark.parametrize("sigma_p2", [1e-2, 3e-4, 1.06e-5])
@pytest.mark.parametrize("n,m,gen", [(9001, 5201, "surface"), (8300, 7500, "cube"), (7307, 9801, "cube"),
                                     (20001, 16300, "surface"), (6200, 50001, "surface")])
def test_local_estep_moments(cesa, oracle, torch_cuda, n, m, gen, sigma_p2):
    from cuda_emicp_softassign_gb300 import workloads as W
    if gen == "cube":
        X, Y, R, t = W.uniform_pair(n=n, m=m, seed=n + m)
    else:
        X, Y, R, t = W.surface_pair(n=n, m=m, seed=n + m, max_deg=20.0, outlier_frac=0.05)
    p = cesa.Params.default(sigma_p2=sigma_p2, sigma_inf=0.09 * sigma_p2)  # 23 steps
    assert cesa.emicp_form(n, m, p) == cesa.EMICP_FORM_LOCAL
    _, _, trace, _ = cesa.emicp(X, Y, R, t, param=p, trace=True)
    rec = trace[0]
    ref = oracle.emicp_step(X, Y, R.astype(np.float32), t.astype(np.float32), sigma_p2, p.d_02)
    extent = float(np.ptp(X, 0).max())
    assert abs(rec[2] - ref["sum"]) <= 1e-5 * ref["sum"]
    assert np.abs(rec[3:6] - ref["Xc"]).max() < 1e-5 * extent
    assert np.abs(rec[6:9] - ref["Yc"]).max() < 1e-5 * extent
    assert rel_err(rec[9:18], ref["S"]) < 1e-5


@pytest.mark.parametrize("n,m", [(9001, 5201), (20001, 16300)])
def test_local_gradients_follow_the_rows(cesa, torch_cuda, n, m):
    """The same cloud in another order of its rows: the same pose, and the gradients
    in that order (a row's is about 1/m of their sum, so one that went astray is off
    by its own size; rounding leaves 1e-5)."""
    from cuda_emicp_softassign_gb300 import workloads as W
    from cuda_emicp_softassign_gb300.autograd import emicp_autograd
    torch = torch_cuda
    X, Y, Rt, _ = W.surface_pair(n=n, m=m, seed=3, max_deg=20.0, outlier_frac=0.05)
    p = cesa.Params.default(sigma_inf=1.5e-3)
    assert cesa.emicp_form(n, m, p) == cesa.EMICP_FORM_LOCAL
    order = np.random.default_rng(1).permutation(m)
    out = []
    for rows in (np.arange(m), order):
        f32 = dict(dtype=torch.float32, device="cuda")
        x, y = torch.tensor(X, requires_grad=True, **f32), torch.tensor(Y[rows], requires_grad=True, **f32)
        R, t = emicp_autograd(x, y, torch.eye(3, **f32), torch.zeros(3, **f32), p)
        loss = ((R - torch.tensor(Rt, **f32)) ** 2).sum() + (t ** 2).sum()
        gx, gy = torch.autograd.grad(loss, (x, y))
        out.append([v.detach().cpu().numpy().astype(np.float64) for v in (R, t, gx, gy)])
    (Ra, ta, gxa, gya), (Rb, tb, gxb, gyb) = out
    assert np.abs(Ra - Rb).max() < 1e-5 and np.abs(ta - tb).max() < 1e-5
    assert rel_err(gxb, gxa) < 1e-4
    assert rel_err(gyb, gya[order]) < 1e-4


@pytest.mark.parametrize("case", ["same", "line", "nan", "inf"])
def test_local_on_degenerate_clouds(cesa, torch_cuda, case):
    """Coincident and collinear points sort and sweep; a coordinate that is not
    finite gives a pose that is not finite in the same places as with direct differences."""
    def run(n, form):
        rng = np.random.default_rng(3)
        X = rng.uniform(0, 0.2, (n, 3)).astype(np.float32)
        Y = X.copy()
        if case == "same":
            Y[:] = Y[0]
        elif case == "line":
            Y[:, 1:] = 0.1
        else:
            Y[7, 2] = np.float32(case)
        p = cesa.Params.default(sigma_inf=1.8e-3)
        assert cesa.emicp_form(n, n, p) == form
        return cesa.emicp(X, Y, param=p)
    (R1, t1), (R2, t2) = run(9000, cesa.EMICP_FORM_LOCAL), run(4800, cesa.EMICP_FORM_ROWS)
    assert np.array_equal(np.isfinite(R1), np.isfinite(R2)) and np.array_equal(np.isfinite(t1), np.isfinite(t2))


def test_ranges_registration(cesa, oracle, torch_cuda):
    """A registration by ranges of tasks (X scaled anew for every step): the pose after
    each step against the FP64 oracle's, 1e-3 degrees and 1e-5 of the extent."""
    from conftest import rot_err_deg
    from cuda_emicp_softassign_gb300 import workloads as W
    X, Y, _, _ = W.surface_pair(n=1025, m=330001, seed=4, max_deg=10.0, outlier_frac=0.05)
    sched = dict(sigma_p2=0.01, sigma_inf=0.0045)  # 8 steps
    p = cesa.Params.default(**sched)
    assert cesa.emicp_form(1025, 330001, p) == cesa.EMICP_FORM_RANGES
    _, _, trace, _ = cesa.emicp(X, Y, param=p, trace=True)
    _, _, ref = oracle.emicp(X, Y, **sched)
    assert len(trace) == len(ref) == 8
    extent = float(np.ptp(X, 0).max())
    for got, want in zip(trace, ref):
        assert rot_err_deg(got[18:27].reshape(3, 3), want[18:27].reshape(3, 3)) < 1e-3
        assert np.abs(got[27:30] - want[27:30]).max() < 1e-5 * extent
