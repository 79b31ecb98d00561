"""Order of the centred SPLIT sweeps: the particles' stable Morton order.

The sums of a centred sweep depend on which particles share a tile and on
their order in it, so a sweep of particles that already stand in that order
(formed here in NumPy) equals, bit for bit, the sweep of the shuffled ones.
Clumped positions make many equal keys, whose order a sort must keep.  Sizes
lie around a block's keys and around the block limit of the sort.
"""

import numpy as np
import pytest

from tupan_gb300 import abi, ics, lib

pytestmark = pytest.mark.gpu


def morton_order(*sets):
    """Stable Morton order of the first set on the grid of all of them."""
    pos = [np.stack([s[k] for k in ("rx", "ry", "rz")]) for s in sets]
    f = np.concatenate(pos, axis=1).astype(np.float32).astype(np.float64)
    lo = f.min(axis=1)
    ext = (f.max(axis=1) - lo).max()
    scale = 65535.0 / ext if ext > 0 else 0.0
    q = np.clip((pos[0] - lo[:, None]) * scale, 0.0, 65535.0)
    q = q.astype(np.uint64)
    key = np.zeros(q.shape[1], dtype=np.uint64)
    for b in range(16):
        for d in range(3):
            bit = (q[d] >> np.uint64(b)) & np.uint64(1)
            key |= bit << np.uint64(3 * b + d)
    return np.argsort(key, kind="stable")


def take(ps, idx):
    return {k: np.ascontiguousarray(v[idx]) for k, v in ps.items()}


def run(name, ips, jps):
    vals = abi.make_args(name, "float64", ips, jps)
    abi.call(lib.bind(name), name, "float64", vals)
    lib.check()
    return abi.outputs(name, vals)


def particles(n, clumped, seed):
    ps = ics.plummer(n, eps=1e-2, seed=seed)
    if clumped:
        for k in ("rx", "ry", "rz"):
            ps[k] = np.round(ps[k] * 8) / 8
    return ps


@pytest.mark.parametrize("clumped", [False, True])
@pytest.mark.parametrize("ni,nj", [(1, 0), (2, 511), (511, 513), (513, 0),
                                   (65536, 300), (300, 65537), (131073, 0)])
def test_shuffled_equals_morton_ordered(ni, nj, clumped):
    ip = particles(ni, clumped, 5)
    jp = particles(nj, clumped, 6) if nj else ip
    sets = (ip, jp) if nj else (ip,)
    oi = morton_order(*sets)
    oj = morton_order(*sets[::-1])
    old = lib.set_mode(lib.MODE_SPLIT)
    lib.set_centred(1, -1, 0)
    try:
        for name in ("phi_kernel", "acc_jerk_kernel"):
            got = run(name, ip, jp)
            si = take(ip, oi)
            want = run(name, si, take(jp, oj) if nj else si)
            for g, w in zip(got, want):
                np.testing.assert_array_equal(g[oi], w, err_msg=name)
    finally:
        lib.set_mode(old)
        lib.set_centred(-1, -1, 0)
