"""GPU: row slices (SBB_KERNEL_SLICED) and the automatic choice that takes
short, even rows to them, against the accurate (double-double) oracle."""
import numpy as np
import pytest

import oracle as O
from helpers import TOL_FP64, max_scaled_err, rand_csr

pytestmark = pytest.mark.gpu

# Slices of 32/W rows: row counts around them; row lengths around W steps, the
# 4 steps in flight and the 1,024 nnz that the plan's copy stages at a time.
MATS = {
    "one_row": lambda: rand_csr(1, 1, 50, 17, 17),
    "31_rows": lambda: rand_csr(2, 31, 300, 0, 9),
    "33_rows": lambda: rand_csr(3, 33, 300, 1, 16),
    "even": lambda: rand_csr(4, 1000, 700, 12, 12),
    "ragged": lambda: rand_csr(5, 1237, 900, 0, 37, p_empty=0.3),
    "long": lambda: rand_csr(6, 97, 3000, 1, 130, long_rows=[(0, 1100), (96, 33)]),
    "one_column": lambda: rand_csr(7, 200, 1, 0, 1),
    "all_empty": lambda: rand_csr(8, 70, 5, 0, 0),
}


def _run(mat, f32, cfg, scal):
    import torch
    from sbb.device import Plan
    rp, col, val, x, y = mat
    d, vt = torch.device("cuda:0"), torch.float32 if f32 else torch.float64
    P = Plan(torch.from_numpy(rp.astype(np.int32)).to(d), torch.from_numpy(col).to(d),
             torch.from_numpy(val).to(d, vt), len(x), f32=f32, **cfg)
    info, outs = P.info(), []
    for alpha, beta in scal:
        yy = torch.from_numpy(y).to(d)
        if beta == 0.0:
            yy.fill_(float("nan"))  # y is not read
        P.spmv(torch.from_numpy(x).to(d, vt), yy, alpha, beta)
        torch.cuda.synchronize()
        outs.append(yy.cpu().numpy())
    P.check()
    P.close()
    return outs, info


@pytest.mark.parametrize("width", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("f32", [False, True], ids=["f64", "f32"])
@pytest.mark.parametrize("name", list(MATS))
def test_sliced_matches_oracle(cuda, name, f32, width):
    rp, col, val, x, y = MATS[name]()
    if f32:
        val, x = val.astype(np.float32).astype(np.float64), x.astype(np.float32).astype(np.float64)
    scal = ((1.0, 0.0), (-0.7, 0.3), (0.0, 2.0))
    outs, info = _run((rp, col, val, x, y), f32, dict(kernel="sliced", vector_width=width), scal)
    assert info["kernel"] == 6 and info["vector_width"] == width
    for (alpha, beta), out in zip(scal, outs):
        ref, sc = O.spmv_dd(rp, col, val, x, alpha, beta, y)
        assert max_scaled_err(out, ref, sc) <= TOL_FP64, (alpha, beta)


@pytest.mark.parametrize("lo,hi,sliced", [(1, 8, True), (24, 24, True), (100, 200, True),
                                          (0, 1, True), (1, 600, False)])
def test_auto_takes_even_rows_to_slices(cuda, lo, hi, sliced):
    """The automatic choice against the merge path on the same matrix."""
    mat = rand_csr(lo + hi, 700, 900, lo, hi,
                   long_rows=[] if sliced else [(r, 2) for r in range(650)])
    (a,), info = _run(mat, False, dict(kernel="auto"), ((1.5, -0.5),))
    (b,), _ = _run(mat, False, dict(kernel="merge"), ((1.5, -0.5),))
    assert (info["kernel"] == 6) == sliced
    _, sc = O.spmv_dd(*mat[:4], 1.5, -0.5, mat[4])
    assert max_scaled_err(a, b, sc) <= 2 * TOL_FP64


def test_auto_with_bad_column_runs_and_reports(cuda):
    """Even rows with a column out of range: the automatic choice needs no copy
    of such a matrix to be refused; it runs and sbb_plan_check reports it, as
    the vector kernel does."""
    import torch
    from sbb.device import Plan, SbbError
    rp, col, val, x, y = rand_csr(9, 500, 400, 4, 8)
    col = col.copy()
    col[77] = len(x)
    d = torch.device("cuda:0")
    P = Plan(torch.from_numpy(rp.astype(np.int32)).to(d), torch.from_numpy(col).to(d),
             torch.from_numpy(val).to(d), len(x))
    assert P.info()["kernel"] == 1
    P.spmv(torch.from_numpy(x).to(d), torch.from_numpy(y).to(d))
    with pytest.raises(SbbError):
        P.check()
    P.close()
    with pytest.raises(SbbError):
        Plan(torch.from_numpy(rp.astype(np.int32)).to(d), torch.from_numpy(col).to(d),
             torch.from_numpy(val).to(d), len(x), kernel="sliced")


def test_sliced_refuses_odd_widths(cuda):
    import torch
    from sbb.device import Plan, SbbError
    z = torch.zeros(3, dtype=torch.int32, device="cuda")
    for w in (3, 32, -1):
        with pytest.raises(SbbError):
            Plan(z, z[:0], torch.zeros(0, dtype=torch.float64, device="cuda"), 4, kernel="sliced",
                 vector_width=w)
