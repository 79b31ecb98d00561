"""SPLIT variants 3 and 4 in packed pairs (many i) and scalar (few i): the
sums of an i do not depend on which ran, so a sweep of many i and one of a
few of them agree bit for bit; and the packed ones stay on the oracle."""

import numpy as np
import pytest

import oracle
from tupan_gb300 import abi, ics, lib

pytestmark = pytest.mark.gpu

KERNELS = {"phi_kernel": None, "acc_kernel": None, "acc_jerk_kernel": None,
           "tstep_kernel": {"eta": 1.0 / 64}, "snap_crackle_kernel": None}


def particles(n, mixed):
    ps = ics.plummer(n, eps=1e-2, seed=61)
    rng = np.random.default_rng(62)
    for k in ("ax", "ay", "az", "jx", "jy", "jz"):
        ps[k] = rng.standard_normal(n)
    if mixed:
        ps["e2"] = ps["e2"] * rng.choice([1.0, 4.0], n)
    return ps


def run(name, ips, jps):
    vals = abi.make_args(name, "float64", ips, jps, KERNELS[name])
    abi.call(lib.bind(name), name, "float64", vals)
    lib.check()
    return abi.outputs(name, vals)


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("variant,gsplit,ni,nj", [
    (3, 1, 3201, 4097), (3, 2, 1601, 2560), (3, 7, 460, 1793),
    (4, 1, 2001, 1300), (4, 2, 1003, 2817), (4, 3, 700, 3329)])
def test_many_i_equal_few_i(variant, gsplit, ni, nj, mixed):
    js = particles(nj, mixed)
    pick = np.arange(ni) % nj
    ips = {k: np.ascontiguousarray(v[pick]) for k, v in js.items()}
    few = [0, 1, 7, ni // 2, ni - 2, ni - 1]
    fps = {k: np.ascontiguousarray(v[few]) for k, v in ips.items()}
    old = lib.set_mode(lib.MODE_SPLIT)
    try:
        for name in KERNELS:
            lib.set_split_config(name, variant, gsplit)
            many = run(name, ips, js)
            part = run(name, fps, js)
            lib.set_split_config(name, -1, 0)
            for m, p in zip(many, part):
                np.testing.assert_array_equal(m[few], p, err_msg=name)
            want = oracle.run(name, fps, js, KERNELS[name])
            for p, w in zip(part, want):
                # FP32 pairs: far below a lost or doubled record (1e-3)
                assert np.abs(p - w).max() <= 1e-4 * np.abs(w).max(), name
    finally:
        lib.set_mode(old)
        for name in KERNELS:
            lib.set_split_config(name, -1, 0)
