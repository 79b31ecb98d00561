"""The workspace that the queued Sakura sweep keeps between calls."""

import numpy as np
import pytest

from tupan_gb300 import ics, lib
from tupan_gb300 import kepler as kp

pytestmark = pytest.mark.gpu
NAMES = ("m", "rx", "ry", "rz", "e2", "vx", "vy", "vz")


def system(n, seed):
    torch = pytest.importorskip("torch")
    ps = ics.plummer(n, eps=0.0, seed=seed, masses="salpeter")
    return ({k: torch.from_numpy(np.ascontiguousarray(ps[k])).cuda()
             for k in NAMES},
            [torch.zeros(n, dtype=torch.float64, device="cuda")
             for _ in range(6)])


def sweep(d, out, n, mode="exact", stream=None):
    ptr = [d[k].data_ptr() for k in NAMES]
    return kp.sakura_queue(n, ptr, n, ptr, [o.data_ptr() for o in out],
                           1.0 / 512, -1, mode=mode, stream=stream)[0]


@pytest.mark.parametrize("mode", ["exact", "split"])
def test_a_sweep_after_one_too_large_for_the_memory(mode):
    n = 257
    d, out = system(n, 21)
    nk = sweep(d, out, n, mode)
    want = [o.cpu().numpy() for o in out]
    # counts of 2^40 particles (4 TiB) cannot be had: refused before any
    # launch or access
    ptr = [d[k].data_ptr() for k in NAMES]
    with pytest.raises(lib.TupanGB300Error, match="status 1"):
        kp.sakura_queue(1 << 40, ptr, 1, ptr, [o.data_ptr() for o in out],
                        1.0 / 512, -1, mode=mode)
    for m in (n, 2 * n):            # the counts fit the old size; grow again
        d, out = system(m, 21)
        for o in out:
            o.fill_(float("nan"))
        got = sweep(d, out, m, mode)
        if m == n:
            assert got == nk
            for o, w in zip(out, want):
                np.testing.assert_array_equal(o.cpu().numpy(), w)
        else:
            assert all(np.isfinite(o.cpu().numpy()).all() for o in out)
