"""The sizes that the no-allocation EM-ICP call takes in its fixed scratch: those that it
took before rows were sorted (the last argument, within 2000 points of what it took
then), and a schedule that sorts them (csrc/cesa_emicp.cu's local form) up to the
sizes of a single step, which does not."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,took", [(0, 129, 1023060), (129, 0, 462951), (1000, 0, 310620), (5000, 0, 293043),
                                      (20000, 0, 280154), (0, 20000, 315307)])
def test_sorted_schedules_take_the_same_sizes(cesa, torch_cuda, n, m, took):
    """(0: the size whose limit is looked for, to the point)"""
    torch = torch_cuda
    cloud = torch.rand(3 * 1100000, device="cuda") * 0.2
    rt = torch.tensor([1, 0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0], dtype=torch.float32, device="cuda")
    step = cesa.Params.default(sigma_inf=0.0095)
    schedule = cesa.Params.default()

    def takes(k, p):
        rc = cesa.emicp_device_noalloc(cloud[:3 * (n or k)], cloud[:3 * (m or k)], rt.clone(), p)
        torch.cuda.synchronize()
        assert rc in (cesa.CESA_OK, cesa.CESA_ERR_NOALLOC_LIMIT)
        return rc == cesa.CESA_OK

    lo, hi = 1000, 1100000
    assert takes(lo, step) and not takes(hi, step)
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (mid, hi) if takes(mid, step) else (lo, mid)
    assert lo >= took and takes(lo, schedule), lo
    status = torch.full((1,), -1, dtype=torch.int32, device="cuda")
    assert cesa.emicp_device_noalloc(cloud[:3 * (n or lo)], cloud[:3 * (m or lo)], rt, schedule,
                                     d_status=status) == cesa.CESA_OK
    torch.cuda.synchronize()
    assert int(status.item()) == cesa.CESA_OK
