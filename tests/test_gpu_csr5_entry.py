"""GPU: csr5_kernel, one product on device pointers, against the accurate
(double-double) oracle; malformed matrices are refused with y untouched."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
from helpers import TOL_FP64, max_scaled_err, rand_csr

pytestmark = pytest.mark.gpu

MATS = {
    "even_6": lambda: rand_csr(1, 1500, 700, 3, 9),
    "even_100": lambda: rand_csr(2, 333, 900, 80, 120),
    "uneven": lambda: rand_csr(3, 2000, 5000, 0, 20, p_empty=0.3, long_rows=[(5, 4000), (1999, 900)]),
    "one_row": lambda: rand_csr(4, 1, 9000, 8000, 8000),
    "no_nnz": lambda: rand_csr(5, 70, 10, 0, 0),
}


def _call(m, n, nnz, alpha, val, rp, col, x, beta, y):
    from sbb import lib
    a, b = C.c_double(alpha), C.c_double(beta)
    return lib().csr5_kernel(m, n, nnz, C.byref(a), val.data_ptr(), rp.data_ptr(), col.data_ptr(),
                             x.data_ptr(), C.byref(b), y.data_ptr())


@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-0.7, 0.3), (0.0, 2.0)])
@pytest.mark.parametrize("name", list(MATS))
def test_csr5_entry_matches_oracle(cuda, name, alpha, beta):
    import torch
    rp, col, val, x, y = MATS[name]()
    d = [torch.from_numpy(a).cuda() for a in (val, rp.astype(np.int32), col, x, y)]
    if beta == 0.0:
        d[4].fill_(float("nan"))  # y is not read
    assert _call(len(y), len(x), len(col), alpha, *d[:4], beta, d[4]) == 0
    got = d[4].cpu().numpy()  # the call has ended when it returns
    ref, sc = O.spmv_dd(rp, col, val, x, alpha, beta, y)
    assert max_scaled_err(got, ref, sc) <= TOL_FP64


@pytest.mark.parametrize("fault", ["column", "negative", "monotone", "first", "last"])
def test_csr5_entry_refuses(cuda, fault):
    import torch
    rp, col, val, x, y = MATS["uneven"]()
    rp, col = rp.astype(np.int32), col.copy()
    if fault == "column":
        col[-1] = len(x)
    elif fault == "negative":
        col[7] = -1
    elif fault == "monotone":
        rp[100] = rp[101] + 1
    elif fault == "first":
        rp[0] = 1
    else:
        rp[-1] -= 1
    d = [torch.from_numpy(a).cuda() for a in (val, rp, col, x, y)]
    assert _call(len(y), len(x), len(col), 1.0, *d[:4], 0.5, d[4]) == -1
    assert np.array_equal(d[4].cpu().numpy(), y)
