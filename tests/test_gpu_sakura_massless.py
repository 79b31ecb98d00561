"""Branch test of the queued Sakura sweep for pairs without mass: the
reference's r^2 > (64 m / v^2)^2 is false where m / v^2 is 0 / 0, so the pair
counts as a Kepler pair."""

import numpy as np
import pytest

from tupan_gb300 import kepler as kp

pytestmark = pytest.mark.gpu
NAMES = ("m", "rx", "ry", "rz", "e2", "vx", "vy", "vz")


def kepler_pairs(ps, dt, flag):
    """Pairs that do not take the leapfrog branch, with numpy."""
    d = {k: ps[k][:, None] - ps[k][None, :] for k in NAMES[1:]}
    if flag == -1:
        for c in "xyz":
            d["r" + c] = d["r" + c] - d["v" + c] * dt
    m = ps["m"][:, None] + ps["m"][None, :]
    r2 = d["rx"] ** 2 + d["ry"] ** 2 + d["rz"] ** 2
    v2 = d["vx"] ** 2 + d["vy"] ** 2 + d["vz"] ** 2
    with np.errstate(divide="ignore", invalid="ignore"):
        R = 64.0 * (m / v2)
        return int(np.sum(~(r2 > R * R)))


@pytest.mark.parametrize("mode", ["exact", "split"])
@pytest.mark.parametrize("flag", [-1, 1])
@pytest.mark.parametrize("n,massless,moving", [
    (1, 1, 0), (6, 6, 0), (6, 4, 1), (40, 33, 20), (300, 200, 1),
    (40, 0, 0)])
def test_massless_pairs_at_relative_rest(n, massless, moving, flag, mode):
    torch = pytest.importorskip("torch")
    ps = {k: np.zeros(n) for k in NAMES}
    ps["rx"] = np.arange(n) * 0.5
    ps["m"][massless:] = 0.25 / n
    ps["vx"][n - moving:] = np.arange(moving) + 1.0
    dt = 1.0 / 512
    d = {k: torch.from_numpy(ps[k]).cuda() for k in NAMES}
    ptr = [d[k].data_ptr() for k in NAMES]
    out = [torch.zeros(n, dtype=torch.float64, device="cuda")
           for _ in range(6)]
    nk, hist = kp.sakura_queue(n, ptr, n, ptr, [o.data_ptr() for o in out],
                               dt, flag, histogram=True, mode=mode)
    assert nk == kepler_pairs(ps, dt, flag) and hist.sum() == nk
