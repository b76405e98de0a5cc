"""Device calls recorded in a CUDA graph: replays on other inputs in the same buffers give
what the call itself gives, bitwise. A batch and the Softassign backward send tables
that the host frees after the call; a graph has to hold them itself."""
import numpy as np
import pytest
from conftest import soa_tensor

pytestmark = pytest.mark.gpu


def _clouds(torch, n, m, seed):
    from cuda_emicp_softassign_gb300 import workloads as W
    X, Y, _, _ = W.surface_pair(n=n, m=m, seed=seed, max_deg=20.0, outlier_frac=0.05)
    return soa_tensor(torch, X), soa_tensor(torch, Y)


def _start(torch):
    return torch.tensor([1, 0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0], dtype=torch.float32, device="cuda")


def _replays(torch, call, buffers, inputs, start):
    """call(buffers) once on the stream for the workspaces and per input for the expected
    results, then recorded, then replayed on every input."""
    s = torch.cuda.Stream()

    def load(given):
        for b, g in zip(buffers, given):
            b.copy_(g)
        for b in buffers[len(given):]:
            b.copy_(start)
        torch.cuda.synchronize()

    want = []
    for given in inputs:
        load(given)
        call(s)
        torch.cuda.synchronize()
        want.append([b.clone() for b in buffers[len(given):]])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        call(s)
    junk = [np.random.default_rng(k).standard_normal(5000) for k in range(200)]  # reuses what the host freed
    for k in (0, 1, 0):
        load(inputs[k])
        graph.replay()
        torch.cuda.synchronize()
        got = [b for b in buffers[len(inputs[k]):]]
        assert all(torch.equal(a, b) for a, b in zip(got, want[k])), k
    assert len(junk) == 200


@pytest.mark.parametrize("name,n,m", [("emicp", 1007, 900), ("emicp", 9001, 9001), ("emicp", 600, 400000),
                                      ("softassign", 700, 700), ("icp", 20000, 20000), ("icp", 1000, 1000)])
def test_single_calls(cesa, torch_cuda, name, n, m):
    torch = torch_cuda
    p = cesa.Params.default(JMAX=10)
    inputs = [_clouds(torch, n, m, seed) for seed in (1, 2)]
    X, Y, rt = inputs[0][0].clone(), inputs[0][1].clone(), _start(torch)
    fn = getattr(cesa, name + "_device")
    _replays(torch, lambda s: fn(X, Y, rt, p, stream=s), [X, Y, rt], inputs, _start(torch))


@pytest.mark.parametrize("pairs", [1, 7, 90])
def test_batch(cesa, torch_cuda, pairs):
    torch = torch_cuda
    p = cesa.Params.default(JMAX=6)
    sizes = [(300 + 37 * (k % 9), 300 + 37 * (k % 9) if k % 2 else 250 + 11 * (k % 13)) for k in range(pairs)]
    inputs = [[c for k, (n, m) in enumerate(sizes) for c in _clouds(torch, n, m, 10 * seed + k % 3)]
              for seed in (1, 2)]
    clouds = [c.clone() for c in inputs[0]]
    poses = [_start(torch) for _ in sizes]
    batch = [(cesa.ALGO_SOFTASSIGN if k % 2 else cesa.ALGO_EMICP, clouds[2 * k], clouds[2 * k + 1], poses[k], p)
             for k in range(pairs)]
    _replays(torch, lambda s: cesa.register_batch_device(batch, stream=s), clouds + poses, inputs, _start(torch))


@pytest.mark.parametrize("kind", ["emicp", "softassign"])
def test_gradients(cesa, torch_cuda, kind):
    from cuda_emicp_softassign_gb300 import workloads as W
    from cuda_emicp_softassign_gb300.autograd import emicp_autograd, softassign_autograd
    torch = torch_cuda
    fn = emicp_autograd if kind == "emicp" else softassign_autograd
    p = cesa.Params.default(T_0=0.1, JMAX=4, sigma_inf=2e-3)
    f32 = dict(dtype=torch.float32, device="cuda")
    inputs = [[torch.tensor(c, **f32) for c in W.surface_pair(n=500, m=500, seed=seed, max_deg=20.0)[:2]] for seed in (1, 2)]
    X, Y = (c.clone().requires_grad_(True) for c in inputs[0])
    eye, zero = torch.eye(3, **f32), torch.zeros(3, **f32)

    def step():
        R, t = fn(X, Y, eye, zero, p)
        return torch.autograd.grad(((R - eye) ** 2).sum() + (t ** 2).sum(), (X, Y))

    def load(given):
        with torch.no_grad():
            X.copy_(given[0])
            Y.copy_(given[1])
        torch.cuda.synchronize()

    s = torch.cuda.Stream()
    want = []
    with torch.cuda.stream(s):
        for given in inputs:
            load(given)
            want.append([g.clone() for g in step()])
            torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        got = step()
    for k in (1, 0):
        load(inputs[k])
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want[k]))
