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
