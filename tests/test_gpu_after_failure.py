"""A sweep that could not get its workspace leaves the next one unaffected."""

import ctypes

import numpy as np
import pytest

import oracle
from tupan_gb300 import ics, lib

pytestmark = pytest.mark.gpu
NAMES = ("m", "rx", "ry", "rz", "e2", "vx", "vy", "vz")


@pytest.mark.parametrize("mode", [lib.MODE_EXACT, lib.MODE_SPLIT])
def test_sweep_after_one_too_large_for_the_memory(mode):
    torch = pytest.importorskip("torch")
    n = 400
    ps = ics.plummer(n, eps=1e-3, seed=2)
    d = [torch.from_numpy(np.ascontiguousarray(ps[k])).cuda() for k in NAMES]
    out = [torch.zeros(n, dtype=torch.float64, device="cuda")
           for _ in range(6)]
    VP = ctypes.c_void_p
    ptr = (VP * 8)(*[t.data_ptr() for t in d])
    outs = (VP * 6)(*[o.data_ptr() for o in out])
    L, k = lib.load(), lib.KERNEL_ID["acc_jerk_kernel"]
    # packed records of 2^40 particles (48 TiB): refused before any launch
    assert L.tupan_gb300_dev_sweep(k, lib.MODE_SPLIT, 1 << 40, ptr, 1, ptr,
                                   None, 0, outs, None, 1) == 1
    assert L.tupan_gb300_dev_sweep(k, mode, n, ptr, n, ptr, None, 0, outs,
                                   None, 1) == 0
    want = oracle.run("acc_jerk_kernel", ps, ps)
    for o, w in zip(out, want):
        tol = 1e-5 * np.abs(w).max() if mode == lib.MODE_SPLIT else 0.0
        assert np.abs(o.cpu().numpy() - w).max() <= tol
