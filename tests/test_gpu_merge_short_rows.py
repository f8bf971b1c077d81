"""GPU: the merge path on rows so short that a segment has more than 32 of them
(their ends are brought to shared memory), against the accurate oracle."""
import numpy as np
import pytest

import oracle as O
from helpers import TOL_FP64, max_scaled_err, rand_csr

pytestmark = pytest.mark.gpu

MATS = {
    "empty": lambda: rand_csr(1, 5000, 7, 0, 0),  # a segment is all row ends
    "one_each": lambda: rand_csr(2, 4099, 900, 1, 1),  # half products, half ends
    "0_to_3": lambda: rand_csr(3, 6001, 900, 0, 3, p_empty=0.3),
    "around_32_rows": lambda: rand_csr(4, 3000, 900, 4, 6),
    "mixed": lambda: rand_csr(5, 5003, 4000, 0, 2, long_rows=[(700, 300), (2500, 3000)]),
}


@pytest.mark.parametrize("ipt", [4, 6, 8, 12])
@pytest.mark.parametrize("f32", [False, True], ids=["f64", "f32"])
@pytest.mark.parametrize("name", list(MATS))
def test_merge_short_rows(cuda, name, f32, ipt):
    import torch
    from sbb.device import Plan
    rp, col, val, x, y = MATS[name]()
    if f32:
        val, x = val.astype(np.float32).astype(np.float64), x.astype(np.float32).astype(np.float64)
    vt = torch.float32 if f32 else torch.float64
    for persistent in (0, 1):
        P = Plan(torch.from_numpy(rp.astype(np.int32)).cuda(), torch.from_numpy(col).cuda(),
                 torch.from_numpy(val).to("cuda", vt), len(x), f32=f32, kernel="merge",
                 items_per_thread=ipt, persistent=persistent)
        for alpha, beta in ((1.0, 0.0), (-0.7, 0.3)):
            ref, sc = O.spmv_dd(rp, col, val, x, alpha, beta, y)
            yd = torch.from_numpy(y).cuda()
            if beta == 0.0:
                yd.fill_(float("nan"))
            P.spmv(torch.from_numpy(x).to("cuda", vt), yd, alpha, beta)
            torch.cuda.synchronize()
            assert max_scaled_err(yd.cpu().numpy(), ref, sc) <= TOL_FP64
        P.check()
        P.close()
