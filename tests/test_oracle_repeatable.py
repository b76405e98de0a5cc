"""The oracle's FP32 port gives one result per input, whatever the number of threads
and in every run: tests hold the kernels against twice its error, which on an
ill-conditioned pair (17 points against 33) was anything between 0.004 and 0.13
degrees while the threads' partial sums were added as they came."""
import numpy as np


def test_f32_port_does_not_depend_on_threads(oracle):
    from cuda_emicp_softassign_gb300 import workloads as W
    X, Y, _, _ = W.surface_pair(n=17, m=33, seed=116)
    most = oracle.max_threads()
    out = []
    try:
        for threads in (1, 2, 5, 5, 5, 16, 16):
            oracle.set_threads(threads)
            R, t, _ = oracle.softassign(X, Y, precision="f32", trace=False, JMAX=8, I0=2, T_0=50.0, TFACTOR=0.6)
            out.append(np.concatenate([np.ravel(R), np.ravel(t)]))
    finally:
        oracle.set_threads(most)
    assert all(np.array_equal(o, out[0]) for o in out)
