"""The wait limit of the centred sweep's tile ring bounds a tile's copy, not
the other warps' work: a low limit does not refuse a sweep whose warps come to
a stage before the slowest one has left it."""

import numpy as np
import pytest

from tupan_gb300 import ics, lib

pytestmark = pytest.mark.gpu
NAMES = ("m", "rx", "ry", "rz", "e2", "vx", "vy", "vz")


# a Plummer sphere: a block's warps see tiles of different classes, so of
# different work; 46400 bodies are many tiles a block, 3000 few
@pytest.mark.parametrize("kernel,na,no", [("phi_kernel", 5, 1),
                                          ("acc_kernel", 5, 3),
                                          ("acc_jerk_kernel", 8, 6)])
@pytest.mark.parametrize("n,shape,gsplit", [(46400, -1, 0), (46400, 2, 1),
                                            (3000, 0, 4)])
def test_low_limit_gives_the_results_of_the_full_one(kernel, na, no, n, shape,
                                                     gsplit):
    torch = pytest.importorskip("torch")
    ps = ics.plummer(n, eps=1e-4, seed=12)
    d = [torch.from_numpy(np.ascontiguousarray(ps[k])).cuda()
         for k in NAMES[:na]]
    ptr = [t.data_ptr() for t in d]
    lib.set_centred(1, shape, gsplit)
    res = []
    try:
        for limit in (1 << 20, 4):
            out = [torch.full((n,), float("nan"), dtype=torch.float64,
                              device="cuda") for _ in range(no)]
            old = lib.set_pipe_spin_limit(limit)
            try:
                for _ in range(3):
                    lib.dev_sweep(kernel, n, ptr, n, ptr,
                                  [o.data_ptr() for o in out],
                                  mode=lib.MODE_SPLIT, sync=True)
            finally:
                lib.set_pipe_spin_limit(old)
            res.append([o.cpu().numpy() for o in out])
    finally:
        lib.set_centred(-1, -1, 0)
    for a, b in zip(*res):
        np.testing.assert_array_equal(b, a)
