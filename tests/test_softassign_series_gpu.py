"""The series form of the Softassign updates (csrc/cesa_softassign_series.cu):
under AUTO the updates whose affinities a short series represents run in one
cluster, and the affinity kernels take the schedule up where it stops.

Tolerance: as for the other forms, a final rotation within 1e-3 degrees of the
FP64 oracle or, where the pair is ill-conditioned, no further from it than
twice the reference's FP32 arithmetic (the oracle's f32 port); translation
within 1e-5 of the extent or twice the port's."""
import numpy as np
import pytest

from conftest import rot_err_deg

pytestmark = pytest.mark.gpu


def _pair(n, m, seed, scale=1.0, shift=0.0):
    from cuda_emicp_softassign_gb300 import workloads as W
    X, Y, _, _ = W.surface_pair(n=n, m=m, seed=seed)
    f = lambda P: (P * np.float32(scale) + np.float32(shift)).astype(np.float32)  # noqa: E731
    return f(X), f(Y)


def _check(cesa, oracle, X, Y, **sched):
    R, t = cesa.softassign(X, Y, param=cesa.Params.default(**sched))
    Ro, to, _ = oracle.softassign(X, Y, trace=False, **sched)
    Rp, tp, _ = oracle.softassign(X, Y, precision="f32", trace=False, **sched)
    ext = float(np.ptp(X, 0).max())
    assert rot_err_deg(R, Ro) <= max(1e-3, 2 * rot_err_deg(Rp, Ro))
    assert np.abs(t - to).max() <= max(1e-5 * ext, 2 * np.abs(tp - to).max())


# edges of the warps (32), of the cluster sizes (128, 256, 512, ... points a
# CTA) and of the uneven last CTA; degrees 2-4
@pytest.mark.parametrize("n,m", [(17, 33), (127, 129), (255, 257), (512, 512), (513, 500), (1025, 1024), (2049, 2048),
                                 (4097, 300), (300, 4097)])
def test_sizes(cesa, oracle, n, m):
    X, Y = _pair(n, m, n + 3 * m)
    _check(cesa, oracle, X, Y, JMAX=8, I0=2, T_0=50.0, TFACTOR=0.6)


# one degree after the other, 2 to 8, and past the last one (the affinity
# kernels' part of the schedule); I1 = 1 and 5 as well
@pytest.mark.parametrize("T0,I1", [(40.0, 3), (3.0, 1), (0.8, 5), (0.4, 3), (0.2, 3), (0.12, 3), (0.08, 3), (0.05, 3)])
def test_degrees(cesa, oracle, T0, I1):
    X, Y = _pair(700, 650, 5)
    _check(cesa, oracle, X, Y, JMAX=3, I0=2, I1=I1, T_0=T0, TFACTOR=0.9)


@pytest.mark.parametrize("n,m", [(600, 600), (1500, 1500)])
def test_hands_over_in_mid_schedule(cesa, oracle, n, m):
    """Clouds of unit extent: the series covers the first temperatures only."""
    X, Y = _pair(n, m, 7, scale=5.0)
    _check(cesa, oracle, X, Y, JMAX=40, TFACTOR=0.88)


def test_off_the_origin(cesa, oracle):
    """Five extents off (the centring offsets are not zero). Softassign's S
    depends on the frame: a hundred off, the FP64 oracle itself ends in NaN."""
    X, Y = _pair(400, 400, 9, shift=1.0)
    _check(cesa, oracle, X, Y, JMAX=20, TFACTOR=0.8)


@pytest.mark.parametrize("case", ["large", "offset", "nan", "inf"])
def test_outside_its_range_the_affinity_kernel_runs_alone(cesa, case):
    """Bitwise the matrix-free form's result: extents of 200, a start 100 apart,
    a coordinate that is not finite."""
    X, Y = _pair(300, 280, 11, scale=1000.0 if case == "large" else 1.0)
    t0 = np.full(3, 60.0) if case == "offset" else np.zeros(3)
    if case in ("nan", "inf"):
        X[5, 1] = np.float32(case)
    sched = dict(JMAX=3)
    a = cesa.softassign(X, Y, t=t0, param=cesa.Params.default(**sched))
    b = cesa.softassign(X, Y, t=t0, param=cesa.Params.default(sinkhorn_form=cesa.SINKHORN_MATRIX_FREE, **sched))
    assert np.array_equal(a[0], b[0], equal_nan=True) and np.array_equal(a[1], b[1], equal_nan=True)


def test_batch_takes_up_where_the_series_stops(cesa):
    """Pairs that run wholly, partly and not at all in the series, beside
    EM-ICP: within 2e-3 degrees of single calls (the batch's own tolerance)."""
    sched = dict(JMAX=30, TFACTOR=0.85)
    pairs = [(cesa.ALGO_SOFTASSIGN, *_pair(300, 300, 1), cesa.Params.default(**sched)),
             (cesa.ALGO_EMICP, *_pair(500, 400, 2), cesa.Params.default()),
             (cesa.ALGO_SOFTASSIGN, *_pair(500, 500, 3, scale=5.0), cesa.Params.default(**sched)),
             (cesa.ALGO_SOFTASSIGN, *_pair(200, 200, 4, scale=100.0), cesa.Params.default(JMAX=3))]
    for (algo, X, Y, p), (R, t) in zip(pairs, cesa.register_batch(pairs)):
        Rs, ts = (cesa.softassign if algo == cesa.ALGO_SOFTASSIGN else cesa.emicp)(X, Y, param=p)
        assert rot_err_deg(R, Rs) < 2e-3
        assert np.abs(t - ts).max() < 1e-4 * float(np.ptp(X, 0).max())


@pytest.mark.parametrize("sizes", [[33, 257, 1025], [513] * 40 + [1535, 1536, 1537, 3073, 24001],
                                   [20011, 16385, 16384, 12289] * 3 + [129] * 30])
def test_batches_of_several_cluster_sizes(cesa, sizes):
    """All clusters at once with few, more and most points per CTA, and more
    clusters than fit: the pairs agree with single calls, both in the series
    (its sums in another order), within the batch's tolerance."""
    p = cesa.Params.default(JMAX=12)
    pairs = [(cesa.ALGO_SOFTASSIGN, *_pair(n, n, k % 7), p) for k, n in enumerate(sizes)]
    single = {}
    for (_, X, Y, _), (R, t), key in zip(pairs, cesa.register_batch(pairs), [(n, k % 7) for k, n in enumerate(sizes)]):
        if key not in single:
            single[key] = cesa.softassign(X, Y, param=p)
        Rs, ts = single[key]
        assert rot_err_deg(R, Rs) < 2e-3
        assert np.abs(t - ts).max() < 1e-4 * float(np.ptp(X, 0).max())
