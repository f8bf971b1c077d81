"""GPU: the automatic choice on matrices with many more rows than nnz."""
import numpy as np
import pytest

import oracle as O
from helpers import TOL_FP64, max_scaled_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,filled,long", [(32_768, 900, 77), (32_769, 900, 77),
                                           (3_000_000, 99_000, 1000), (40_000_000, 500, 500)])
def test_nearly_empty_matrices(cuda, m, filled, long):
    """`filled` rows of one nnz and one long row between empty ones, first and
    last row among the filled: row pieces up to 32,768 rows, tiles above."""
    import torch
    from sbb.device import Plan
    rng = np.random.default_rng(m)
    at = np.sort(rng.choice(np.arange(1, m - 1), filled, replace=False))
    lens = np.zeros(m, np.int64)
    lens[at] = 1
    lens[[0, m - 1]] = 2
    lens[m // 2] = long
    rp = np.concatenate([[0], np.cumsum(lens)])
    n = 5000
    col = rng.integers(0, n, rp[-1]).astype(np.int32)
    val, x, y = rng.uniform(-1, 1, rp[-1]), rng.uniform(-1, 1, n), rng.uniform(-1, 1, m)
    P = Plan(torch.from_numpy(rp.astype(np.int32)).cuda(), torch.from_numpy(col).cuda(),
             torch.from_numpy(val).cuda(), n)
    info = P.info()
    assert info["kernel"] == (7 if m <= 32_768 else 3)
    assert info["scratch_bytes"] <= 32 * m + 100 * rp[-1] + (1 << 20)
    yd = torch.from_numpy(y).cuda()
    P.spmv(torch.from_numpy(x).cuda(), yd, 1.5, -0.5)
    torch.cuda.synchronize()
    P.check()
    P.close()
    got = yd.cpu().numpy()
    full = np.flatnonzero(lens)  # the oracle on the filled rows; the others are beta * y
    ref, sc = O.spmv_dd(np.concatenate([[0], np.cumsum(lens[full])]), col, val, x, 1.5, -0.5, y[full])
    assert max_scaled_err(got[full], ref, sc) <= TOL_FP64
    got[full] = -0.5 * y[full]
    assert np.array_equal(got, -0.5 * y)
