"""i and j records packed in one launch: sizes around a block of the packing
kernel and beyond the blocks that it launches at most."""

import numpy as np
import pytest

import oracle
from tupan_gb300 import abi, ics, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ni,nj", [(1, 1), (63, 65), (64, 64), (65, 129),
                                   (3, 650001), (650001, 3)])
@pytest.mark.parametrize("name", ["acc_kernel", "acc_jerk_kernel",
                                  "snap_crackle_kernel"])
def test_both_sets(name, ni, nj):
    ps = ics.plummer(ni + nj, eps=1e-2, seed=17)
    rng = np.random.default_rng(18)
    for k in ("ax", "ay", "az", "jx", "jy", "jz"):
        ps[k] = rng.standard_normal(ni + nj)
    ip = {k: np.ascontiguousarray(v[:ni]) for k, v in ps.items()}
    jp = {k: np.ascontiguousarray(v[ni:]) for k, v in ps.items()}
    old = lib.set_mode(lib.MODE_SPLIT)
    try:
        vals = abi.make_args(name, "float64", ip, jp)
        abi.call(lib.bind(name), name, "float64", vals)
        lib.check()
        got = abi.outputs(name, vals)
    finally:
        lib.set_mode(old)
    want = oracle.run(name, ip, jp)
    for c in range(0, len(want), 3):
        # FP32 pair terms (1e-6) whose parts cancel up to a hundredfold; an
        # unpacked or misplaced record gives another particle's term
        scale = max(np.abs(w).max() for w in want[c:c + 3])
        for g, w in zip(got[c:c + 3], want[c:c + 3]):
            assert np.abs(g - w).max() <= 1e-4 * scale, name
