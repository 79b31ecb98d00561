"""The reduction of grid j-split partial sums at the edges of its shape (32 i
a block, eight groups of splits) against the fp64 oracle."""

import numpy as np
import pytest

import oracle
from tupan_gb300 import abi, ics, lib

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def spheres():
    js = ics.plummer(17000, eps=1e-3, seed=21)
    cut = {n: {k: np.ascontiguousarray(v[:n]) for k, v in js.items()}
           for n in (1, 31, 33, 65)}
    want = {n: (oracle.run("acc_jerk_kernel", cut[n], js),
                oracle.run("tstep_kernel", cut[n], js, {"eta": 1.0 / 64}))
            for n in cut}
    return js, cut, want


@pytest.mark.parametrize("gsplit", [2, 7, 8, 9, 16, 17, 63, 64])
@pytest.mark.parametrize("ni", [1, 31, 33, 65])
def test_partials_reduced_like_the_oracle(spheres, ni, gsplit):
    js, cut, want = spheres
    got = {}
    old = lib.set_mode(lib.MODE_SPLIT)
    try:
        for name, sc in (("acc_jerk_kernel", None),
                         ("tstep_kernel", {"eta": 1.0 / 64})):
            lib.set_split_config(name, 4, gsplit)
            vals = abi.make_args(name, "float64", cut[ni], js, sc)
            abi.call(lib.bind(name), name, "float64", vals)
            lib.check()
            got[name] = abi.outputs(name, vals)
    finally:
        lib.set_mode(old)
        for name in ("acc_jerk_kernel", "tstep_kernel"):
            lib.set_split_config(name, -1, 0)
    # FP32 pairs summed to 2^-48: 1e-5 of the largest value is a hundred
    # rounding errors, a lost or doubled split changes it by 1/gsplit
    for g, w in zip(got["acc_jerk_kernel"] + got["tstep_kernel"],
                    want[ni][0] + want[ni][1]):
        assert np.abs(g - w).max() <= 1e-5 * np.abs(w).max()
