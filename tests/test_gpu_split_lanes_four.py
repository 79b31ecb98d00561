"""Packed pairs on four lanes an i (variant 6): the lanes' sums of the scalar
form on four lanes (variant 2), up to the rounding of FP32 pairs, at the edges
of a block's 128 i and of a tile."""

import numpy as np
import pytest

import oracle
from tupan_gb300 import abi, ics, lib

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sphere():
    return ics.plummer(2900, eps=1e-3, seed=31)


@pytest.mark.parametrize("kernel,scal", [("phi_kernel", None),
                                         ("acc_jerk_kernel", None),
                                         ("tstep_kernel", {"eta": 1.0 / 64})])
@pytest.mark.parametrize("ni", [1, 2, 127, 129, 1025])
@pytest.mark.parametrize("gsplit", [1, 3])
def test_four_lanes(sphere, kernel, scal, ni, gsplit):
    ips = {k: np.ascontiguousarray(v[:ni]) for k, v in sphere.items()}
    want = oracle.run(kernel, ips, sphere, scal)
    old = lib.set_mode(lib.MODE_SPLIT)
    try:
        for variant in (2, 6):
            lib.set_split_config(kernel, variant, gsplit)
            vals = abi.make_args(kernel, "float64", ips, sphere, scal)
            abi.call(lib.bind(kernel), kernel, "float64", vals)
            lib.check()
            # FP32 pairs summed to 2^-48: 1e-5 of the largest value is a
            # hundred rounding errors, a lane lost or counted twice a quarter
            for g, w in zip(abi.outputs(kernel, vals), want):
                assert np.abs(g - w).max() <= 1e-5 * np.abs(w).max()
    finally:
        lib.set_mode(old)
        lib.set_split_config(kernel, -1, 0)
