"""GPU: the automatic choice goes on without the row slices' copy when that does
not fit (the device allocation really fails: the armed hook asks for more than
any device has), and the failure does not come back as an error of a product."""
import numpy as np
import pytest

import oracle as O
from helpers import TOL_FP64, max_scaled_err, rand_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [2, 3])  # 1: the plan's status words; then the copy's two arrays
def test_vector_kernel_when_the_copy_does_not_fit(cuda, k):
    import torch
    from sbb._lib import TEST_FAIL_ALLOC, TEST_RESET, lib
    from sbb.device import Plan
    rp, col, val, x, y = rand_csr(21, 3001, 900, 4, 9)
    a = (torch.from_numpy(rp.astype(np.int32)).cuda(), torch.from_numpy(col).cuda(),
         torch.from_numpy(val).cuda())
    dx, dy = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    lib().sbb_test_hook(TEST_FAIL_ALLOC, k)
    try:
        P = Plan(*a, len(x))
    finally:
        lib().sbb_test_hook(TEST_RESET, 0)
    assert P.info()["kernel"] == 1
    P.spmv(dx, dy, 1.5, -0.5)
    torch.cuda.synchronize()
    P.check()
    P.close()
    ref, sc = O.spmv_dd(rp, col, val, x, 1.5, -0.5, y)
    assert max_scaled_err(dy.cpu().numpy(), ref, sc) <= TOL_FP64
    P = Plan(*a, len(x))
    assert P.info()["kernel"] == 6
    P.close()


@pytest.mark.parametrize("k", [2, 3, 4, 5])  # the counters, the list, the sums, the counts of rows
def test_row_pieces_without_memory(cuda, k):
    """A list that does not fit is refused, and the next plan is as any other."""
    import torch
    from sbb._lib import TEST_FAIL_ALLOC, TEST_RESET, lib
    from sbb.device import Plan, SbbError
    rp, col, val, x, y = rand_csr(22, 300, 900, 0, 9, long_rows=[(7, 700)])
    a = (torch.from_numpy(rp.astype(np.int32)).cuda(), torch.from_numpy(col).cuda(),
         torch.from_numpy(val).cuda())
    lib().sbb_test_hook(TEST_FAIL_ALLOC, k)
    try:
        with pytest.raises(SbbError):
            Plan(*a, len(x))
    finally:
        lib().sbb_test_hook(TEST_RESET, 0)
    P = Plan(*a, len(x))
    assert P.info()["kernel"] == 7
    dy = torch.from_numpy(y).cuda()
    P.spmv(torch.from_numpy(x).cuda(), dy, 1.5, -0.5)
    torch.cuda.synchronize()
    P.close()
    ref, sc = O.spmv_dd(rp, col, val, x, 1.5, -0.5, y)
    assert max_scaled_err(dy.cpu().numpy(), ref, sc) <= TOL_FP64
