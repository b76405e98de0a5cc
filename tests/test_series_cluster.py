"""The cluster of the Softassign series form (csrc/cesa_softassign_series.cu) where the device
holds only smaller ones, or none: never larger than that, and the affinity kernels
alone (0) where the points do not fit it. Host arithmetic, needs no GPU."""
import pytest


@pytest.mark.parametrize("most", [16, 8, 4, 2, 1, 0])
def test_never_larger_than_the_device_holds(cesa, most):
    fn = cesa.lib().cesa_self_test_series_cluster
    for n, m in [(1, 1), (413, 413), (2000, 2000), (7001, 6007), (300, 4097), (20000, 20000), (30000, 30000)]:
        got = fn(n, m, most)
        assert got <= most
        assert got == 0 or got & (got - 1) == 0
        full = fn(n, m, 16)
        assert got in (0, min(full, most))
        if most == 0:
            assert got == 0


def test_sizes(cesa):
    fn = cesa.lib().cesa_self_test_series_cluster
    assert [fn(n, n, 16) for n in (100, 413, 2000, 20000, 30000)] == [1, 4, 8, 16, 0]
    assert [fn(n, n, 1) for n in (100, 1000, 2000)] == [1, 1, 0]
    assert fn(20000, 20000, 8) == 0
    assert fn(0, 5, 16) == 0 and fn(5, 1 << 24, 16) == 0
