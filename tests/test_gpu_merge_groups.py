"""GPU: merge-path segments taken several to a warp (matrices that make at least
eight waves of blocks), against the oracle and, bit for bit, against the
persistent form, which claims other numbers of segments."""
import numpy as np
import pytest

import oracle as O
from helpers import TOL_FP64, max_scaled_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ipt", [4, 6, 12])
@pytest.mark.parametrize("m,lmax,p_empty", [(700_001, 18, 0.1), (2_500_003, 2, 0.5),
                                            (9_973, 900, 0.0)])
def test_merge_groups(cuda, m, lmax, p_empty, ipt):
    import torch
    from sbb.device import Plan
    rng = np.random.default_rng(m)
    lens = rng.integers(0, lmax + 1, m)
    lens[rng.random(m) < p_empty] = 0
    lens[m // 2] = 70_000
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    n = 50_000
    col = rng.integers(0, n, rp[-1]).astype(np.int32)
    val, x, y = rng.uniform(-1, 1, rp[-1]), rng.uniform(-1, 1, n), rng.uniform(-1, 1, m)
    d = [torch.from_numpy(a).cuda() for a in (rp.astype(np.int32), col, val)]
    outs = []
    for persistent in (0, 2):
        P = Plan(*d, n, kernel="merge", items_per_thread=ipt, persistent=persistent)
        yy = torch.from_numpy(y).cuda()
        P.spmv(torch.from_numpy(x).cuda(), yy, 1.25, -0.5)
        torch.cuda.synchronize()
        P.check()
        P.close()
        outs.append(yy.cpu().numpy())
    assert np.array_equal(outs[0], outs[1])
    ref, sc = O.spmv_dd(rp, col, val, x, 1.25, -0.5, y)
    assert max_scaled_err(outs[0], ref, sc) <= TOL_FP64
