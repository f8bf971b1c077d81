"""GPU: the sizes that row pieces are cut in: rows that would have more pieces than
one warp adds, rows that are one piece each, rows that finish in one warp, and
the lanes that the automatic choice takes on small matrices."""
import numpy as np
import pytest

import oracle as O
from helpers import TOL_FP64, max_scaled_err, rand_csr

pytestmark = pytest.mark.gpu


def _rows(seed, lens, n):
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    return (rp, rng.integers(0, n, rp[-1]).astype(np.int32), rng.uniform(-1, 1, rp[-1]),
            rng.uniform(-1, 1, n), rng.uniform(-1, 1, len(lens)))


MATS = {  # lengths, width, pieces
    "200k_8": (lambda: [3, 200_001, 0, 70], 8, None),  # 1,024 pieces of a row at most
    "100k_8": (lambda: [100_000] * 4 + [64, 65], 8, None),
    "2.5M_32": (lambda: [5, 2_500_000, 1], 32, None),  # 2,048 of a row at most
    "single": (lambda: np.random.default_rng(1).integers(300, 2018, 7000), 32, 7000),
    "finish_together": (lambda: np.random.default_rng(2).integers(60, 200, 3001), 8, None),
}


@pytest.mark.parametrize("f32", [False, True], ids=["f64", "f32"])
@pytest.mark.parametrize("name", list(MATS))
def test_piece_sizes(cuda, name, f32):
    import torch
    from sbb.device import Plan
    lens, width, pieces = MATS[name]
    rp, col, val, x, y = _rows(3, np.asarray(lens()), 30_011)
    if f32:
        val, x = val.astype(np.float32).astype(np.float64), x.astype(np.float32).astype(np.float64)
    vt = torch.float32 if f32 else torch.float64
    ref, sc = O.spmv_dd(rp, col, val, x, 1.5, -0.5, y)
    outs = []
    for _ in range(2):  # two plans: their lists are numbered in different orders
        P = Plan(torch.from_numpy(rp.astype(np.int32)).cuda(), torch.from_numpy(col).cuda(),
                 torch.from_numpy(val).to("cuda", vt), len(x), f32=f32, kernel="pieces",
                 vector_width=width)
        assert pieces is None or P.info()["tiles"] == pieces
        for _ in range(2):
            yd = torch.from_numpy(y).cuda()
            P.spmv(torch.from_numpy(x).to("cuda", vt), yd, 1.5, -0.5)
            torch.cuda.synchronize()
            outs.append(yd.cpu().numpy())
        P.check()
        P.close()
    assert max_scaled_err(outs[0], ref, sc) <= TOL_FP64
    assert all(np.array_equal(outs[0], o) for o in outs[1:])


@pytest.mark.parametrize("lens,width", [([1000] * 100, 32), ([131_072], 32), ([1000, 24] * 50, 32),
                                        ([1000, 22] * 50, 8), ([1] * 900 + [1000], 8)])
def test_lanes_on_small_matrices(cuda, lens, width):
    import torch
    from sbb.device import Plan
    rp, col, val, x, y = _rows(4, np.asarray(lens), 9_001)
    P = Plan(torch.from_numpy(rp.astype(np.int32)).cuda(), torch.from_numpy(col).cuda(),
             torch.from_numpy(val).cuda(), len(x))
    i = P.info()
    yd = torch.from_numpy(y).cuda()
    P.spmv(torch.from_numpy(x).cuda(), yd, 1.5, -0.5)
    torch.cuda.synchronize()
    P.close()
    assert (i["kernel"], i["vector_width"]) == (7, width)
    ref, sc = O.spmv_dd(rp, col, val, x, 1.5, -0.5, y)
    assert max_scaled_err(yd.cpu().numpy(), ref, sc) <= TOL_FP64


def test_no_rows(cuda):
    import torch
    from sbb.device import Plan
    z = torch.zeros(1, dtype=torch.int32, device="cuda")
    P = Plan(z, z[:0], torch.zeros(0, dtype=torch.float64, device="cuda"), 4)
    y = torch.zeros(0, dtype=torch.float64, device="cuda")
    P.spmv(torch.zeros(4, dtype=torch.float64, device="cuda"), y, 1.0, 0.0)
    torch.cuda.synchronize()
    P.check()
    P.close()
