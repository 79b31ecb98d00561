"""Block shapes and queue growth of the EXACT queued Sakura sweep, against
the oracle."""

import numpy as np
import pytest

import oracle
from tupan_gb300 import ics
from tupan_gb300 import kepler as kp

pytestmark = pytest.mark.gpu
NAMES = ("m", "rx", "ry", "rz", "e2", "vx", "vy", "vz")


def check(ips, jps, dt, flag):
    torch = pytest.importorskip("torch")
    ni, nj = len(ips["m"]), len(jps["m"])
    dev = [[torch.from_numpy(np.ascontiguousarray(p[k])).cuda()
            for k in NAMES] for p in (ips, jps)]
    out = [torch.zeros(ni, dtype=torch.float64, device="cuda")
           for _ in range(6)]
    nk, hist = kp.sakura_queue(ni, [t.data_ptr() for t in dev[0]], nj,
                               [t.data_ptr() for t in dev[1]],
                               [o.data_ptr() for o in out], dt, flag,
                               histogram=True)
    torch.cuda.synchronize()
    assert hist.sum() == nk
    want = oracle.run("sakura_kernel", ips, jps, {"dt": dt, "flag": flag})
    for c in range(6):
        keys = NAMES[1:4] if c < 3 else NAMES[5:]
        scale = max(np.abs(p[k]).max() for p in (ips, jps) for k in keys)
        # the bound test_sakura_queue_matches_oracle holds the sweep to
        assert np.abs(out[c].cpu().numpy() - want[c]).max() <= 1e-12 * scale
    return nk


# i counts either side of each change of the i's a block (600 << k)
@pytest.mark.parametrize("flag", [-1, 1])
@pytest.mark.parametrize("ni,nj", [(1, 300), (599, 129), (1201, 65),
                                   (2403, 31), (4801, 17), (9601, 9)])
def test_block_shapes(ni, nj, flag):
    check(ics.plummer(ni, eps=0.0, seed=8, masses="salpeter"),
          ics.plummer(nj, eps=0.0, seed=9, masses="salpeter"), 1.0 / 512,
          flag)


def test_queue_grows_when_most_pairs_are_kepler():
    # slow bodies: every pair takes the Kepler branch, more than the 2^20
    # entries a first queue has at most
    ps = ics.plummer(1100, eps=0.0, seed=10)
    for k in ("vx", "vy", "vz"):
        ps[k] *= 1e-3
    assert check(ps, ps, 1.0 / 4096, -1) == 1100 * 1100
