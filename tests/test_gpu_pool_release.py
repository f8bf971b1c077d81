"""GPU: what the library's pool holds beyond its bound is back with the device
when a plan, a batch or a tuning run has ended, and get_gpu_availble_mem counts
what the pool holds within the bound as free."""
import pytest

pytestmark = pytest.mark.gpu

SLACK = 256 << 20  # contexts, modules and the rounding of the device's pages


def _even(nnz, per_row):
    """nnz / per_row rows of per_row nnz in one column, all zeros."""
    import torch
    m = nnz // per_row
    rp = torch.arange(0, (m + 1) * per_row, per_row, dtype=torch.int32, device="cuda")
    return (rp, torch.zeros(m * per_row, dtype=torch.int32, device="cuda"),
            torch.zeros(m * per_row, dtype=torch.float64, device="cuda"))


@pytest.mark.parametrize("what", ["plan", "batch", "tune"])
def test_nothing_above_the_bound_is_kept(cuda, what):
    import torch
    from sbb.batch import Batch, tune
    from sbb.device import Plan
    total = torch.cuda.mem_get_info(0)[1]
    rp, col, val = _even(3 * (total // 32) // 12, 64)  # tiles: three times the bound
    m = rp.numel() - 1
    x, y = (torch.zeros(k, dtype=torch.float64, device="cuda") for k in (4, m))
    d = dict(m=m, n=4, rowptr=rp, col=col, val=val, x=x, y=y, alpha=1.0, beta=0.0)
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info(0)[0]
    if what == "plan":
        P = Plan(rp, col, val, 4, kernel="tiled")
        P.close()
    elif what == "batch":
        B = Batch([d], [5])
        B.close()
    else:
        tune(d, reps=1)
    free1 = torch.cuda.mem_get_info(0)[0]
    del rp, col, val, x, y, d
    torch.cuda.empty_cache()
    assert free0 - free1 <= total // 32 + SLACK


def test_available_memory_counts_what_the_pool_holds(cuda):
    import torch
    from sbb import api
    from sbb.device import Plan
    total = torch.cuda.mem_get_info(0)[1]
    rp, col, val = _even(total // 64 // 12, 64)  # a plan of half the bound
    torch.cuda.synchronize()
    before = api.get_gpu_availble_mem(1)
    P = Plan(rp, col, val, 4, kernel="tiled")
    P.close()
    assert api.get_gpu_availble_mem(1) >= before - SLACK / 1e9
    P = Plan(rp, col, val, 4, kernel="tiled")
    P.close()
    torch.cuda.synchronize()  # and given back
    assert api.get_gpu_availble_mem(1) >= before - SLACK / 1e9
    assert torch.cuda.mem_get_info(0)[0] / 1e9 >= before - SLACK / 1e9
