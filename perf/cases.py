"""Performance cases: what a user of this framework has it do.

Every case is one pass through the public Python API of
cuda_emicp_softassign_gb300 on seeded synthetic scans: two partly overlapping
views of a union of ellipsoids (workloads.surface_pair), the stand-in for the
scan pairs that this kind of registration is run on, with the sizes of the
repository's benchmark configurations and odd, ragged ones between them.

  emicp            one EM-ICP registration of device clouds, default schedule
  emicp_host       the same from host arrays, copies included
  emicp_grad       EM-ICP forward and backward: the pose of a differentiable
                   registration and the gradients of a pose loss in both clouds
  softassign       one Softassign registration of device clouds
  softassign_host  the same from host arrays
  softassign_grad  Softassign forward and backward
  batch            many uneven pairs in one call, EM-ICP and Softassign mixed
  icp              ICP with the default nearest-neighbour search
"""
import math

import numpy as np
import torch
import torch.utils.checkpoint

import cuda_emicp_softassign_gb300 as cesa
from cuda_emicp_softassign_gb300 import workloads
from cuda_emicp_softassign_gb300.autograd import emicp_autograd, softassign_autograd

DEV = "cuda"


def listed():
    return [
        # the smallest call: a scan thinned to about a thousand points, from host arrays (latency)
        {"name": "emicp_host_1007", "kind": "emicp_host", "n": 1007, "m": 1007},
        # an ordinary pair of unequal, odd sizes, already on the device
        {"name": "emicp_8171x6007", "kind": "emicp", "n": 8171, "m": 6007},
        # full scans: the benchmark's default workload
        {"name": "emicp_40097", "kind": "emicp", "n": 40097, "m": 40097},
        # a training step through the registration
        {"name": "emicp_grad_10007x9001", "kind": "emicp_grad", "n": 10007, "m": 9001},
        # Softassign on heavily thinned scans, from host arrays
        {"name": "softassign_host_413", "kind": "softassign_host", "n": 413, "m": 413},
        # Softassign on scans thinned to 5%, the usual size for it
        {"name": "softassign_2000", "kind": "softassign", "n": 2000, "m": 2000},
        # a ragged pair, refined over the last part of the schedule
        {"name": "softassign_7001x6007_T0.1", "kind": "softassign", "n": 7001, "m": 6007, "T_0": 0.1, "JMAX": 6},
        # unthinned scans
        {"name": "softassign_20000", "kind": "softassign", "n": 20000, "m": 20000},
        # a training step through 30 unrolled pose updates
        {"name": "softassign_grad_2003_T0.1", "kind": "softassign_grad", "n": 2003, "m": 2003, "T_0": 0.1, "JMAX": 6},
        # a set of scan pairs registered together
        {"name": "batch_40", "kind": "batch", "pairs": 40, "lo": 500, "hi": 20000},
        # full scans, rigid ICP
        {"name": "icp_40097", "kind": "icp", "n": 40097, "m": 40097},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Sizes over the logarithm of each kind's range. Softassign runs its
    default schedule on clouds of equal counts, and on unequal counts (or in a
    training step) a schedule that starts at a lower temperature: the default
    one keeps the assignment of unequal clouds so near to uniform that rounding
    decides the pose."""
    kind = rng.choice(["emicp", "emicp", "emicp_host", "emicp_grad", "softassign", "softassign", "softassign_host",
                       "softassign_grad", "batch", "icp"])
    if kind == "batch":
        return {"kind": kind, "pairs": rng.randint(4, 40), "lo": 500, "hi": _log_int(rng, 2000, 16000)}
    lo, hi = {"emicp": (1000, 40000), "emicp_host": (1000, 40000), "emicp_grad": (1000, 20000),
              "softassign": (400, 16000), "softassign_host": (400, 16000), "softassign_grad": (400, 8000),
              "icp": (1000, 40000)}[kind]
    n = _log_int(rng, lo, hi)
    m = min(hi, max(lo, int(round(n * math.exp(rng.uniform(-0.25, 0.25))))))
    case = {"kind": kind, "n": n, "m": m}
    if kind == "softassign_grad":
        case.update(m=n, T_0=0.1, JMAX=rng.randint(3, 8))
    elif kind.startswith("softassign"):
        if rng.random() < 0.6:
            case.update(m=n)
        else:
            case.update(T_0=0.1, JMAX=rng.randint(4, 8))
    return case


def _is_soft(kind):
    return kind.startswith("softassign")


def _clouds(kind, n, m, seed):
    """One scan pair: X (target), Y (source), the true rotation and translation."""
    if _is_soft(kind):  # two views 45 degrees apart
        return workloads.surface_pair(n=n, m=m, seed=seed)
    # views up to 20 degrees apart with 5% of stray points
    return workloads.surface_pair(n=n, m=m, seed=seed, max_deg=20.0, outlier_frac=0.05)


def _params(case):
    return cesa.Params.default(**{k: case[k] for k in ("JMAX", "T_0") if k in case})


def _soa(P):
    return torch.from_numpy(np.ascontiguousarray(P.T).reshape(-1)).to(DEV)


def _start():
    return torch.tensor([1, 0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0], dtype=torch.float32, device=DEV)


def _batch_pairs(case, seed):
    """Sizes log-uniform in [lo, hi], every second pair Softassign (equal counts)."""
    rng = np.random.default_rng(seed)
    out = []
    for k in range(case["pairs"]):
        n, m = (int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]))))) for _ in range(2))
        kind = "softassign" if k % 2 else "emicp"
        m = n if k % 2 else m
        X, Y, _, _ = _clouds(kind, n, m, int(rng.integers(1 << 31)))
        out.append((kind, X, Y))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        p = _params(case)
        q = cesa.Params.default(JMAX=60)
        s = {"kind": kind, "start": _start(), "pairs": []}
        for k, X, Y in _batch_pairs(case, seed):
            soft = k == "softassign"
            s["pairs"].append((cesa.ALGO_SOFTASSIGN if soft else cesa.ALGO_EMICP, _soa(X), _soa(Y), _start(),
                               q if soft else p))
        return s
    X, Y, Rt, tt = _clouds(kind, case["n"], case["m"], seed)
    s = {"kind": kind, "param": _params(case)}
    if kind.endswith("_host"):
        s.update(X=X, Y=Y)
    elif kind.endswith("_grad"):
        f32 = dict(dtype=torch.float32, device=DEV)
        s.update(X=torch.tensor(X, requires_grad=True, **f32), Y=torch.tensor(Y, requires_grad=True, **f32),
                 R0=torch.eye(3, **f32), t0=torch.zeros(3, **f32), Rt=torch.tensor(Rt, **f32),
                 tt=torch.tensor(tt, **f32))
    else:
        s.update(X=_soa(X), Y=_soa(Y), start=_start(), rt=_start())
    return s


def run(s):
    kind = s["kind"]
    if kind == "batch":
        for _, _, _, rt, _ in s["pairs"]:
            rt.copy_(s["start"])
        cesa.register_batch_device(s["pairs"])
        return torch.stack([rt for _, _, _, rt, _ in s["pairs"]])
    if kind.endswith("_host"):
        R, t = (cesa.emicp if kind == "emicp_host" else cesa.softassign)(s["X"], s["Y"], param=s["param"])
        return R.astype(np.float32), t.astype(np.float32)  # the library's values are float32
    if kind.endswith("_grad"):
        fn = emicp_autograd if kind == "emicp_grad" else softassign_autograd
        R, t = fn(s["X"], s["Y"], s["R0"], s["t0"], s["param"])
        loss = ((R - s["Rt"]) ** 2).sum() + ((t - s["tt"]) ** 2).sum()
        gX, gY = torch.autograd.grad(loss, (s["X"], s["Y"]))
        return R.detach(), t.detach(), gX, gY
    s["rt"].copy_(s["start"])
    fn = {"emicp": cesa.emicp_device, "softassign": cesa.softassign_device, "icp": cesa.icp_device}[kind]
    fn(s["X"], s["Y"], s["rt"], s["param"])
    return s["rt"]


# ---------------------------------------------------------------- work and exact values

def _sigmas(p):
    out, s = [], np.float32(p.sigma_p2)
    while s > np.float32(p.sigma_inf):
        out.append(float(s))
        s = np.float32(s * np.float32(p.sigma_factor))
    return out


def _temps(p):
    out, T = [], np.float32(p.T_0)
    for _ in range(p.JMAX):
        out += [float(T)] * p.I0
        T = np.float32(T * np.float32(p.TFACTOR))
    return out


def _pair_work(kind, n, m, p):
    """Bytes: the clouds once, the pose, the gradients. Operations of the
    defining double sums: an EM-ICP affinity 12 (squared distance 6, exponent
    1, five sums) and its adjoint 19, a Softassign pass 8 and its last one 12,
    an ICP distance 6."""
    io = 12.0 * (n + m) + 96
    if kind.startswith("emicp"):
        ops = float(n) * m * len(_sigmas(p)) * (31 if kind.endswith("_grad") else 12)
    elif kind.startswith("softassign"):
        per = 2 * p.I1 * 8 + 12
        ops = float(n) * m * p.JMAX * p.I0 * (per * (2.2 if kind.endswith("_grad") else 1))
    else:
        ops = float(n) * m * p.maxIteration * 6
    return io * (2 if kind.endswith("_grad") else 1), ops


def work(case):
    p = _params(case)
    if case["kind"] == "batch":
        q = cesa.Params.default(JMAX=60)
        # expected sizes of the log-uniform draw
        lo, hi, ln = case["lo"], case["hi"], math.log(case["hi"] / case["lo"])
        mean, rms = (hi - lo) / ln, math.sqrt((hi * hi - lo * lo) / (2 * ln))
        b = o = 0.0
        for k in range(case["pairs"]):
            x, y = _pair_work("softassign", rms, rms, q) if k % 2 else _pair_work("emicp", mean, mean, p)
            b, o = b + x, o + y
        return {"bytes": b, "flops": o}
    b, o = _pair_work(case["kind"], case["n"], case["m"], p)
    return {"bytes": b, "flops": o}


def _horn(S):
    """Horn's 4 x 4 matrix of the cross-covariance S[i, j] = sum x_i y_j."""
    (a, b, c), (d, e, f), (g, h, k) = S[0], S[1], S[2]
    # Sxx = S[0,0], Syx = S[0,1] in the (y, x) naming of Horn's paper
    sxx, sxy, sxz, syx, syy, syz, szx, szy, szz = a, d, g, b, e, h, c, f, k
    return torch.stack([
        torch.stack([sxx + syy + szz, syz - szy, szx - sxz, sxy - syx]),
        torch.stack([syz - szy, sxx - syy - szz, sxy + syx, szx + sxz]),
        torch.stack([szx - sxz, sxy + syx, syy - sxx - szz, syz + szy]),
        torch.stack([sxy - syx, szx + sxz, syz + szy, szz - sxx - syy])])


def _pose(S, Xc, Yc):
    q = torch.linalg.eigh(_horn(S))[1][:, -1]
    w, x, y, z = q
    R = torch.stack([
        torch.stack([w * w + x * x - y * y - z * z, 2 * (x * y - w * z), 2 * (x * z + w * y)]),
        torch.stack([2 * (x * y + w * z), w * w - x * x + y * y - z * z, 2 * (y * z - w * x)]),
        torch.stack([2 * (x * z - w * y), 2 * (y * z + w * x), w * w - x * x - y * y + z * z])])
    return R, Xc - R @ Yc


def _sqdist(A, B):
    """Squared distances of the rows of A and B, centred on B (64-bit)."""
    c = B.detach().mean(0)
    A, B = A - c, B - c
    return ((A * A).sum(1)[:, None] + (B * B).sum(1)[None, :] - 2 * A @ B.T).clamp_min(0)


def _emicp_step(X, Y, R, t, s2, d02):
    Z = Y @ R.T + t
    out = math.exp(-d02 / s2)
    lam, U = [], []
    for Zc in Z.split(max(1, 200_000_000 // len(X))):
        e = torch.exp(_sqdist(Zc, X) * (-0.5 / s2))
        C = (e * e).sum(1) + out
        low = C <= 10e-7
        inv = torch.rsqrt(torch.where(low, torch.ones_like(C), C))
        lam.append(torch.where(low, torch.ones_like(C), e.sum(1) * inv))
        U.append(torch.where(low[:, None], X.mean(0)[None, :], (e @ X) * inv[:, None]))
    lam, U = torch.cat(lam), torch.cat(U)
    L = lam.sum()
    Xc, Yc = U.sum(0) / L, (lam[:, None] * Y).sum(0) / L
    return _pose((U - lam[:, None] * Xc).T @ (Y - Yc), Xc, Yc)


def _emicp64(X, Y, R, t, p, tape=False):
    for s2 in _sigmas(p):
        a = (X, Y, R, t, s2, float(np.float32(p.d_02)))
        R, t = torch.utils.checkpoint.checkpoint(_emicp_step, *a, use_reentrant=False) if tape else _emicp_step(*a)
    return R, t


def _soft_step(X, Y, R, t, s, u, T, p):
    """One pose update, with the assignment as K scaled by row and column vectors."""
    Z = Y @ R.T + t
    K = torch.exp((float(np.float32(p.alpha)) - _sqdist(X, Z)) / T) / math.sqrt(T)
    a, b = torch.ones_like(X[:, 0]), torch.ones_like(Y[:, 0])
    for _ in range(p.I1):
        rs = a * (K @ b) + s
        a, s = a / rs, s / rs
        cs = b * (K.T @ a) + u
        b, u = b / cs, u / cs
    w = a * (K @ b)
    tot = w.sum()
    Xc = (w[:, None] * X).sum(0) / tot
    Yc = (cs[:, None] * Y).sum(0) / tot
    V = a[:, None] * (K @ (b[:, None] * (cs[:, None] * Y - Yc)))
    return (*_pose((w[:, None] * X - Xc).T @ V, Xc, Yc), s, u)


def _soft64(X, Y, R, t, p, tape=False):
    s = torch.full_like(X[:, 0], float(np.float32(p.moutlier)))
    u = torch.full_like(Y[:, 0], float(np.float32(p.moutlier)))
    for T in _temps(p):
        a = (X, Y, R, t, s, u, T, p)
        R, t, s, u = torch.utils.checkpoint.checkpoint(_soft_step, *a, use_reentrant=False) if tape else _soft_step(*a)
    return R, t


def _icp64(X, Y, R, t, p):
    Yc = Y.mean(0)
    for _ in range(p.maxIteration):
        Z = Y @ R.T + t
        nn = torch.cat([_sqdist(Zc, X).argmin(1) for Zc in Z.split(max(1, 200_000_000 // len(X)))])
        Xm = X[nn]
        Xc = Xm.mean(0)
        R, t = _pose((Xm - Xc).T @ (Y - Yc), Xc, Yc)
    return R, t


def exact(case, seed):
    kind = case["kind"]
    f64 = dict(dtype=torch.float64, device=DEV)
    p = _params(case)
    R, t = torch.eye(3, **f64), torch.zeros(3, **f64)
    if kind == "batch":
        if case["pairs"] * case["hi"] ** 2 > 2e9:
            return None
        q = cesa.Params.default(JMAX=60)
        out = []
        for k, X, Y in _batch_pairs(case, seed):
            X, Y = torch.tensor(X, **f64), torch.tensor(Y, **f64)
            Rk, tk = _soft64(X, Y, R, t, q) if k == "softassign" else _emicp64(X, Y, R, t, p)
            out.append(torch.cat([Rk.reshape(-1), tk]))
        return torch.stack(out)
    n, m = case["n"], case["m"]
    if _is_soft(kind) and n * m * p.JMAX > (6e8 if kind.endswith("_grad") else 1.2e10):
        return None
    if kind.endswith("_grad") and n * m > 2e8:
        return None
    X, Y, Rt, tt = _clouds(kind, n, m, seed)
    grad = kind.endswith("_grad")
    X, Y = torch.tensor(X, requires_grad=grad, **f64), torch.tensor(Y, requires_grad=grad, **f64)
    if kind == "icp":
        R, t = _icp64(X, Y, R, t, p)
    elif _is_soft(kind):
        R, t = _soft64(X, Y, R, t, p, tape=grad)
    else:
        R, t = _emicp64(X, Y, R, t, p, tape=grad)
    if grad:
        loss = ((R - torch.tensor(Rt, **f64)) ** 2).sum() + ((t - torch.tensor(tt, **f64)) ** 2).sum()
        gX, gY = torch.autograd.grad(loss, (X, Y))
        return R.detach(), t.detach(), gX, gY
    if kind.endswith("_host"):
        return R, t
    return torch.cat([R.reshape(-1), t])
