"""GPU: rows in pieces (SBB_KERNEL_PIECES) and the automatic choice that takes
long rows to them, against the accurate (double-double) oracle."""
import numpy as np
import pytest

import oracle as O
from helpers import TOL_FP64, max_scaled_err, rand_csr

pytestmark = pytest.mark.gpu

# Lengths around a step (8 or 32), the steps in flight (32 or 128) and a piece (64
# for 8 lanes; 256 for these sizes and 32 lanes, 1,024 from 7.3M nnz); rows that
# start anywhere in their 8 or 32.
MATS = {
    "one": lambda: rand_csr(1, 1, 9000, 7001, 7001),
    "around_a_piece": lambda: rand_csr(2, 200, 2000, 250, 262),
    "around_two": lambda: rand_csr(3, 90, 2000, 480, 545),
    "short_and_empty": lambda: rand_csr(4, 700, 500, 0, 40, p_empty=0.4),
    "around_64": lambda: rand_csr(8, 500, 2000, 55, 75),
    "around_8": lambda: rand_csr(9, 777, 2000, 6, 36, p_empty=0.1),
    "mixed": lambda: rand_csr(5, 300, 70000, 0, 3, long_rows=[(0, 65536), (77, 1023), (299, 33000)]),
    "empty": lambda: rand_csr(6, 33, 5, 0, 0),
    "large": lambda: _large(),
}


def _large():
    rng = np.random.default_rng(7)
    m, n = 5003, 60_000
    lens = rng.integers(900, 2300, m)
    lens[[0, 100, m - 1]] = (0, 400_000, 1)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    return (rp, rng.integers(0, n, rp[-1]).astype(np.int32), rng.uniform(-1, 1, rp[-1]),
            rng.uniform(-1, 1, n), rng.uniform(-1, 1, m))


def _plan(mat, f32, **cfg):
    import torch
    from sbb.device import Plan
    rp, col, val, x, _ = mat
    vt = torch.float32 if f32 else torch.float64
    return Plan(torch.from_numpy(rp.astype(np.int32)).cuda(), torch.from_numpy(col).cuda(),
                torch.from_numpy(val).to("cuda", vt), len(x), f32=f32, **cfg)


@pytest.mark.parametrize("width", [8, 32])
@pytest.mark.parametrize("f32", [False, True], ids=["f64", "f32"])
@pytest.mark.parametrize("name", list(MATS))
def test_pieces_match_oracle(cuda, name, f32, width):
    import torch
    rp, col, val, x, y = MATS[name]()
    if f32:
        val, x = val.astype(np.float32).astype(np.float64), x.astype(np.float32).astype(np.float64)
    P = _plan((rp, col, val, x, y), f32, kernel="pieces", vector_width=width)
    dx = torch.from_numpy(x).to("cuda", torch.float32 if f32 else torch.float64)
    for alpha, beta in ((1.0, 0.0), (-0.7, 0.3)):
        ref, sc = O.spmv_dd(rp, col, val, x, alpha, beta, y)
        outs = []
        for _ in range(3):  # the counts of pieces done come back to zero by themselves
            yy = torch.from_numpy(y).cuda()
            if beta == 0.0:
                yy.fill_(float("nan"))
            P.spmv(dx, yy, alpha, beta)
            torch.cuda.synchronize()
            outs.append(yy.cpu().numpy())
        assert max_scaled_err(outs[0], ref, sc) <= TOL_FP64
        assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[0], outs[2])
    P.check()
    P.close()


def test_auto_takes_long_rows_to_pieces(cuda):
    """Against the merge path on the same matrix; bad columns are refused."""
    import torch
    from sbb.device import SbbError
    mat = MATS["large"]()
    rp, col, val, x, y = mat
    outs = []
    for cfg in (dict(), dict(kernel="merge")):
        P = _plan(mat, False, **cfg)
        assert cfg or P.info()["kernel"] == 7
        yy = torch.from_numpy(y).cuda()
        P.spmv(torch.from_numpy(x).cuda(), yy, 1.5, -0.5)
        torch.cuda.synchronize()
        P.check()
        P.close()
        outs.append(yy.cpu().numpy())
    _, sc = O.spmv_dd(rp, col, val, x, 1.5, -0.5, y)
    assert max_scaled_err(outs[0], outs[1], sc) <= 2 * TOL_FP64
    col[1234] = len(x)
    with pytest.raises(SbbError):
        _plan(mat, False)
    col[1234] = 0
    for mat in (MATS["mixed"](), rand_csr(10, 20_000, 900, 0, 20, long_rows=[(5, 400)])):
        P = _plan(mat, False)  # small and uneven: 8 lanes a piece; larger: the tiles
        info = P.info()
        assert (info["kernel"], info["vector_width"]) == (7, 8) or len(mat[1]) > 1 << 17
        assert info["kernel"] == 3 or len(mat[1]) <= 1 << 17
        P.close()
