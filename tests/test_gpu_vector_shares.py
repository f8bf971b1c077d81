"""GPU: the vector kernel on matrices where a warp takes several chunks of rows
(with FP32 storage that is a kernel of its own), against the accurate oracle."""
import numpy as np
import pytest

import oracle as O
from helpers import TOL_FP64, max_scaled_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f32", [False, True], ids=["f64", "f32"])
@pytest.mark.parametrize("width", [2, 4, 8, 16, 32])
def test_several_chunks_a_warp(cuda, width, f32):
    import torch
    from sbb.device import Plan
    rng = np.random.default_rng(width)
    m, n = 640_007, 5000  # 148 * 32 warps, twice, of chunks of at most 32 rows
    lens = rng.integers(0, 4, m)
    lens[rng.integers(0, m, 500)] = rng.integers(30, 140, 500)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    vt = np.float32 if f32 else np.float64
    col = rng.integers(0, n, rp[-1]).astype(np.int32)
    val, x = rng.uniform(-1, 1, rp[-1]).astype(vt), rng.uniform(-1, 1, n).astype(vt)
    y = rng.uniform(-1, 1, m)
    P = Plan(torch.from_numpy(rp.astype(np.int32)).cuda(), torch.from_numpy(col).cuda(),
             torch.from_numpy(val).cuda(), n, f32=f32, kernel="vector", vector_width=width)
    for alpha, beta in ((1.0, 0.0), (-0.7, 0.3)):
        ref, sc = O.spmv_dd(rp, col, val.astype(np.float64), x.astype(np.float64), alpha, beta, y)
        yd = torch.from_numpy(y).cuda()
        P.spmv(torch.from_numpy(x).cuda(), yd, alpha, beta)
        torch.cuda.synchronize()
        assert max_scaled_err(yd.cpu().numpy(), ref, sc) <= TOL_FP64
    P.check()
    P.close()
