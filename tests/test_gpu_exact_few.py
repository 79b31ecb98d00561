"""EXACT double sweeps of few i (one i a block, sums by warps of their own) at
the edges of a run (128 terms), a tile (256 j) and of the dispatch, with
running sums that cross binades, cancel, tie and overflow: equal bits to the
oracle."""

import numpy as np
import pytest

import oracle
from tupan_gb300 import abi, ics, lib

pytestmark = pytest.mark.gpu

KERNELS = {"phi_kernel": None, "acc_kernel": None, "acc_jerk_kernel": None,
           "snap_crackle_kernel": None, "tstep_kernel": {"eta": 1.0 / 64},
           "nreg_Xkernel": {"dt": 1.0 / 64}, "nreg_Vkernel": {"dt": 1.0 / 64},
           "pnacc_kernel": dict(order=5, **{"inv%d" % k: 128.0 ** -k
                                            for k in range(1, 8)})}


def particles(n, seed):
    ps = ics.plummer(n, eps=1e-2, seed=seed)
    rng = np.random.default_rng(seed)
    for k in ("ax", "ay", "az", "jx", "jy", "jz"):
        ps[k] = rng.standard_normal(n)
    return ps


def check(ips, jps, kernels=KERNELS):
    old = lib.set_mode(lib.MODE_EXACT)
    try:
        for name in kernels:
            vals = abi.make_args(name, "float64", ips, jps, KERNELS[name])
            abi.call(lib.bind(name), name, "float64", vals)
            lib.check()
            want = oracle.run(name, ips, jps, KERNELS[name])
            for got, ref in zip(abi.outputs(name, vals), want):
                np.testing.assert_array_equal(got, ref, err_msg=name)
    finally:
        lib.set_mode(old)


@pytest.mark.parametrize("ni,nj", [(1, 1), (3, 4), (3, 5), (7, 127), (7, 128),
                                   (7, 129), (5, 255), (5, 257), (5, 383),
                                   (2, 1030), (304, 300), (305, 300)])
def test_runs_and_tiles(ni, nj):
    check(particles(ni, 31), particles(nj, 32))


@pytest.mark.parametrize("ni", [5000, 5001])
def test_dispatch_edge_of_one_signed_sums(ni):
    check(particles(ni, 33), particles(40, 34), ("phi_kernel",
                                                 "tstep_kernel"))


@pytest.mark.parametrize("kind", ["powers", "signs", "overflow", "tiny",
                                  "nonfinite", "ties"])
def test_running_sums(kind):
    n = 700
    ips, jps = particles(9, 35), particles(n, 36)
    rng = np.random.default_rng(37)
    if kind == "powers":           # every term another binade
        jps["m"] = 2.0 ** rng.integers(-60, 60, n).astype(float)
    elif kind == "signs":          # sums of both signs through zero
        jps["m"] = rng.standard_normal(n)
    elif kind == "overflow":
        jps["m"] = jps["m"] * 2.0 ** 1019
    elif kind == "tiny":           # subnormal terms and sums
        jps["m"] = jps["m"] * 2.0 ** -1062
    elif kind == "nonfinite":
        jps["m"][300] = np.inf
        jps["m"][500] = -np.inf
    else:                          # equal distances, masses on half grids
        for k in ("rx", "ry", "rz"):
            ips[k][:] = 0.0
            jps[k][:] = 0.0
        jps["rx"][:] = 2.0
        for p in (ips, jps):
            p["e2"][:] = 0.0
        jps["m"] = rng.integers(1, 9, n) * 2.0 ** -rng.integers(
            40, 56, n).astype(float)
        jps["m"][0] = 2.0
    with np.errstate(all="ignore"):
        check(ips, jps)
