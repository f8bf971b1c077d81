"""GPU: a plan reports the shape of the kernel that it has, and no other's."""
import numpy as np
import pytest

from helpers import rand_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel,auto_rows,width", [("sliced", (8, 8), 1), ("pieces", (0, 90), 8),
                                                    ("pieces", (600, 2600), 32)])
def test_info_of_slices_and_pieces(cuda, kernel, auto_rows, width):
    import torch
    from sbb.device import Plan
    rp, col, val, x, y = rand_csr(3, 50 if width == 32 else 300, 3000, *auto_rows,
                                  long_rows=[] if kernel == "sliced" else [(1, 1200)])
    a = (torch.from_numpy(rp.astype(np.int32)).cuda(), torch.from_numpy(col).cuda(),
         torch.from_numpy(val).cuda())
    for cfg in (dict(), dict(kernel=kernel)):
        P = Plan(*a, len(x), **cfg)
        i = P.info()
        assert i["kernel"] == (6 if kernel == "sliced" else 7)
        assert i["vector_width"] in (8, 32) or kernel == "sliced"
        assert cfg or kernel == "sliced" or i["vector_width"] == width
        assert (i["items_per_thread"], i["tile_sigma"], i["persistent"]) == (0, 0, 0)
        P.close()
