"""GPU: the vector kernel's chunks and read-ahead at their edges, standalone and
in a batch, against the accurate (double-double) oracle."""
import numpy as np
import pytest

import oracle as O
from helpers import TOL_FP64, max_scaled_err, rand_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,lo,hi", [(1, 3, 3), (17, 0, 5), (257, 1, 40), (128 * 9 + 5, 0, 8),
                                     (1000, 60, 70), (400, 250, 260)])
@pytest.mark.parametrize("width", [2, 4, 8, 16, 32])
@pytest.mark.parametrize("f32", [False, True], ids=["f64", "f32"])
def test_vector_edges(cuda, m, lo, hi, width, f32):
    """Row counts around a chunk and a warp's share of chunks; rows around the
    lanes and around the 256 nnz of a chunk that are read ahead; arrays that
    start 4 or 8 bytes past a 16-byte boundary and end in their buffer."""
    import torch
    from sbb.device import Plan
    rp, col, val, x, y = rand_csr(m + lo, m, 600, lo, hi, p_empty=0.2 if lo == 0 else 0.0)
    if f32:
        val, x = val.astype(np.float32).astype(np.float64), x.astype(np.float32).astype(np.float64)
    vt = torch.float32 if f32 else torch.float64
    dcol = torch.zeros(len(col) + 1, dtype=torch.int32, device="cuda")[1:]
    dval = torch.zeros(len(col) + 1, dtype=vt, device="cuda")[1:]
    dcol.copy_(torch.from_numpy(col))
    dval.copy_(torch.from_numpy(val))
    P = Plan(torch.from_numpy(rp.astype(np.int32)).cuda(), dcol, dval, len(x), kernel="vector",
             vector_width=width, f32=f32)
    yy = torch.from_numpy(y).cuda()
    P.spmv(torch.from_numpy(x).to("cuda", vt), yy, -0.7, 0.3)
    torch.cuda.synchronize()
    P.check()
    P.close()
    ref, sc = O.spmv_dd(rp, col, val, x, -0.7, 0.3, y)
    assert max_scaled_err(yy.cpu().numpy(), ref, sc) <= TOL_FP64


@pytest.mark.parametrize("count", [1, 7])
def test_batch_vector_classes_at_unit_edges(cuda, count):
    """Matrices of the vector classes around a unit's nnz and rows, and a bad
    column among them: the batch equals the per-matrix launches bit for bit
    and reports the column."""
    import torch
    from sbb.batch import Batch, BatchError
    mats = []
    for k in range(count):
        m = (1, 3, 257, 1000, 33, 64, 2049)[k]
        lo, hi = ((5, 5), (100, 120), (1, 8), (20, 30), (40, 60), (16, 16), (2, 6))[k]
        rp, col, val, x, y = rand_csr(60 + k, m, 500, lo, hi)
        mats.append(dict(m=m, n=500, rp=rp, c=col, v=val, xh=x, yh=y, alpha=-1.25, beta=0.5,
                         rowptr=torch.from_numpy(rp.astype(np.int32)).cuda(),
                         col=torch.from_numpy(col).cuda(), val=torch.from_numpy(val).cuda(),
                         x=torch.from_numpy(x).cuda(), y=torch.from_numpy(y).cuda()))
    B = Batch(mats, [k % 4 for k in range(count)])
    outs = []
    for run in (B.run_each, B.run, B.run_graph):
        for d in mats:
            d["y"].copy_(torch.from_numpy(d["yh"]))
        run()
        torch.cuda.synchronize()
        outs.append([d["y"].cpu().numpy() for d in mats])
    B.check()
    B.close()
    for k, d in enumerate(mats):
        assert np.array_equal(outs[0][k], outs[1][k]) and np.array_equal(outs[0][k], outs[2][k])
        ref, sc = O.spmv_dd(d["rp"], d["c"], d["v"], d["xh"], -1.25, 0.5, d["yh"])
        assert max_scaled_err(outs[1][k], ref, sc) <= TOL_FP64
    mats[0]["col"][0] = -1
    B = Batch(mats, [k % 4 for k in range(count)])
    B.run()
    with pytest.raises(BatchError):
        B.check()
    B.close()
