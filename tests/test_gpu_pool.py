"""GPU: the library's memory pool keeps a bounded amount between calls, leaves
the device's default pool alone, and serves several threads."""
import threading

import numpy as np
import pytest

import oracle as O
from helpers import TOL_FP64, max_scaled_err, rand_csr

pytestmark = pytest.mark.gpu


def test_pool_bounded_and_threads(cuda):
    import torch
    from sbb.device import Plan
    rp, col, val, x, y = rand_csr(3, 3000, 2000, 0, 30, long_rows=[(7, 1500)])
    ref, sc = O.spmv_dd(rp, col, val, x, 1.5, 0.5, y)
    d = torch.device("cuda:0")
    free0, total = torch.cuda.mem_get_info(0)
    out, err = {}, []

    def work(k):
        try:
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                a = (torch.from_numpy(rp.astype(np.int32)).to(d), torch.from_numpy(col).to(d),
                     torch.from_numpy(val).to(d))
                dx, dy = torch.from_numpy(x).to(d), torch.from_numpy(y).to(d)
                for kernel in ("tiled", "merge", "sliced", "rows") * 3:
                    yy = dy.clone()
                    P = Plan(*a, len(x), kernel=kernel)
                    P.spmv(dx, yy, 1.5, 0.5)
                    P.close()
                    out[k, kernel] = yy.cpu().numpy()
        except Exception as e:  # noqa: BLE001
            err.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not err and len(out) == 16
    for v in out.values():
        assert max_scaled_err(v, ref, sc) <= TOL_FP64
    # a plan of a quarter of the bound and more comes and goes: no more than
    # the bound (and what else the process mapped) stays with the library
    n = int(total // 32 // 12)
    z = torch.zeros(2, dtype=torch.int32, device=d)
    z[1] = n
    big = Plan(z, torch.zeros(n, dtype=torch.int32, device=d),
               torch.zeros(n, dtype=torch.float64, device=d), 4, kernel="tiled")
    big.close()
    del big
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    assert free0 - torch.cuda.mem_get_info(0)[0] <= total // 32 + (1 << 30)


CAPTURE = """
import ctypes as C, sys
sys.path.insert(0, sys.argv[1])
import torch
from sbb import lib
rp = torch.tensor([0, 2, 5], dtype=torch.int32, device="cuda")
col = torch.arange(5, dtype=torch.int32, device="cuda")
out, ref = (torch.zeros(12, device="cuda") for _ in range(2))
def call(t, s):
    return lib().sbb_features(2, 5, 5, C.c_void_p(rp.data_ptr()), C.c_void_p(col.data_ptr()),
                              C.c_void_p(t.data_ptr()), C.c_void_p(s.cuda_stream))
s = torch.cuda.Stream()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g, stream=s):  # the library's first allocation
    assert call(out, torch.cuda.current_stream()) == 0
g.replay()
torch.cuda.synchronize()
assert call(ref, torch.cuda.current_stream()) == 0
torch.cuda.synchronize()
assert torch.equal(out, ref) and float(ref.abs().sum()) > 0
"""


def test_first_allocation_inside_a_capture(cuda):
    """A call that allocates stream-ordered scratch, captured in a graph before
    the library has made its pool (in a process of its own)."""
    import os
    import subprocess
    import sys
    import sbb
    pkg = os.path.dirname(os.path.dirname(os.path.abspath(sbb.__file__)))
    r = subprocess.run([sys.executable, "-c", CAPTURE, pkg], capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0, r.stderr[-800:]
