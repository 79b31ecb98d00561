"""EXACT sweeps at the edges of their block shapes (i's a block, pairs a
thread, j's a tile) and on operands the integer-pipe arithmetic hands back
to the FP64 unit: equal bits to the oracle."""

import numpy as np
import pytest

import oracle
from tupan_gb300 import abi, ics, lib

pytestmark = pytest.mark.gpu

KERNELS = ("phi_kernel", "acc_kernel", "acc_jerk_kernel",
           "snap_crackle_kernel", "tstep_kernel", "nreg_Xkernel",
           "nreg_Vkernel")
SCAL = {"tstep_kernel": {"eta": 1.0 / 64}, "nreg_Xkernel": {"dt": 1.0 / 64},
        "nreg_Vkernel": {"dt": 1.0 / 64}}


def particles(n, seed, prec):
    ps = ics.plummer(n, eps=1e-2, seed=seed)
    rng = np.random.default_rng(seed)
    for k in ("ax", "ay", "az", "jx", "jy", "jz"):
        ps[k] = rng.standard_normal(n)
    dt = abi.numpy_real(prec)
    return {k: v.astype(dt) for k, v in ps.items()}


def check(name, ips, jps, prec):
    old = lib.set_mode(lib.MODE_EXACT)
    try:
        fn = lib.bind(name, prec)
        vals = abi.make_args(name, prec, ips, jps, SCAL.get(name))
        abi.call(fn, name, prec, vals)
        lib.check(prec)
    finally:
        lib.set_mode(old)
    want = oracle.run(name, ips, jps, SCAL.get(name), prec=prec)
    for got, ref in zip(abi.outputs(name, vals), want):
        np.testing.assert_array_equal(got, ref, err_msg=name)


# i counts either side of each change of the i's a block (600 << k), j counts
# either side of a tile (a block's 128 threads over its i's)
@pytest.mark.parametrize("prec", ["float64", "float32"])
@pytest.mark.parametrize("ni,nj", [
    (1, 1), (1, 257), (2, 129), (5, 128), (599, 127), (601, 1), (1199, 65),
    (1200, 64), (1203, 63), (2401, 33), (4799, 31), (4801, 17), (9603, 16),
    (19201, 9)])
def test_block_shapes(ni, nj, prec):
    ips, jps = particles(ni, 3, prec), particles(nj, 4, prec)
    for name in KERNELS:
        check(name, ips, jps, prec)


def special(kind, n, prec):
    ps = particles(n, 6, prec)
    rng = np.random.default_rng(7)
    if kind == "planar":
        for k in ("rz", "vz", "az", "jz"):
            ps[k][:] = 0.0
    elif kind == "cold":
        for k in ("vx", "vy", "vz", "ax", "ay", "az", "jx", "jy", "jz"):
            ps[k][:] = 0.0
    elif kind == "lattice":      # coincident bodies, exact and tied roundings
        for k in ("rx", "ry", "rz", "vx", "vy", "vz"):
            ps[k][:] = rng.integers(-3, 4, n) * 0.25
        ps["e2"][:] = rng.choice([0.0, 0.125], n)
    elif kind == "massless":
        ps["m"][rng.random(n) < 0.5] = 0.0
        ps["e2"][:] = 0.0
    elif kind == "scales":       # out of the integer forms' range in places
        big = 2.0 ** (300 if prec == "float64" else 30)
        f = rng.choice([1.0, 1.0 / big, big], n).astype(ps["m"].dtype)
        for k in ps:
            ps[k] = ps[k] * f
    else:
        ps["rx"][::7] = np.inf
        ps["vy"][::11] = np.nan
        ps["m"][::13] = -np.inf
        ps["e2"][::17] = np.nan
    return ps


@pytest.mark.parametrize("prec", ["float64", "float32"])
@pytest.mark.parametrize("kind", ["planar", "cold", "lattice", "massless",
                                  "scales", "nonfinite"])
def test_special_operands(kind, prec):
    ps = special(kind, 333, prec)
    with np.errstate(all="ignore"):
        for name in KERNELS:
            check(name, ps, ps, prec)
