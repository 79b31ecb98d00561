"""SPLIT variants whose lanes share an i: the lanes' sums, added with each lane
keeping a part, for every number of sums (outputs times i a thread) and lanes;
and sums below FP32's normal range, which reach double by another way."""

import numpy as np
import pytest

import oracle
from tupan_gb300 import abi, ics, lib

pytestmark = pytest.mark.gpu

KERNELS = {"phi_kernel": None, "acc_kernel": None, "acc_jerk_kernel": None,
           "tstep_kernel": {"eta": 1.0 / 64}, "snap_crackle_kernel": None}


def run(name, ips, jps):
    vals = abi.make_args(name, "float64", ips, jps, KERNELS[name])
    abi.call(lib.bind(name), name, "float64", vals)
    lib.check()
    return abi.outputs(name, vals)


@pytest.mark.parametrize("variant", [2, 3, 4, 6])
@pytest.mark.parametrize("ni,nj,gsplit", [(1, 2, 1), (5, 700, 1), (33, 700, 3),
                                          (1030, 513, 2), (4001, 300, 1)])
def test_every_output_of_every_lane(variant, ni, nj, gsplit):
    ps = ics.plummer(ni + nj, eps=1e-2, seed=43)
    rng = np.random.default_rng(44)
    for k in ("ax", "ay", "az", "jx", "jy", "jz"):
        ps[k] = rng.standard_normal(ni + nj)
    ip = {k: np.ascontiguousarray(v[:ni]) for k, v in ps.items()}
    jp = {k: np.ascontiguousarray(v[ni:]) for k, v in ps.items()}
    old = lib.set_mode(lib.MODE_SPLIT)
    try:
        for name in KERNELS:
            lib.set_split_config(name, variant, gsplit)
            got = run(name, ip, jp)
            lib.set_split_config(name, -1, 0)
            want = oracle.run(name, ip, jp, KERNELS[name])
            for c in range(0, len(want), 3):
                # FP32 pair terms (1e-6) whose parts cancel up to a
                # hundredfold; a lost or exchanged sum is another i's or
                # axis's
                scale = max(np.abs(w).max() for w in want[c:c + 3])
                for g, w in zip(got[c:c + 3], want[c:c + 3]):
                    assert np.abs(g - w).max() <= 1e-4 * scale, (name, c)
    finally:
        lib.set_mode(old)
        for name in KERNELS:
            lib.set_split_config(name, -1, 0)


@pytest.mark.parametrize("variant", [2, 3, 4, 6])
def test_subnormal_sums(variant):
    # one j of mass 2^-130 at distances of 1 to 9: potentials of 2^-130 and
    # below, exact in FP32 to half its smallest step, and a few roundings
    n = 9
    z = np.zeros(n)
    ip = {"m": np.ones(n), "rx": np.arange(1.0, n + 1), "ry": z, "rz": z,
          "e2": z, "vx": z, "vy": z, "vz": z}
    jp = {k: np.zeros(1) for k in ip}
    jp["m"] = np.array([2.0 ** -130])
    old = lib.set_mode(lib.MODE_SPLIT)
    lib.set_split_config("phi_kernel", variant, 1)
    try:
        got = run("phi_kernel", ip, jp)[0]
    finally:
        lib.set_mode(old)
        lib.set_split_config("phi_kernel", -1, 0)
    want = oracle.run("phi_kernel", ip, jp)[0]
    assert np.abs(got - want).max() <= 4 * 2.0 ** -149
