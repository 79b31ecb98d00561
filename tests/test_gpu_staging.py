"""Host-array calls either side of the pinned staging buffer's limit (1 MiB of
arrays: AccJerk of about 9360 bodies), growing and shrinking between calls:
equal bits to the oracle, inputs untouched."""

import numpy as np
import pytest

import oracle
from tupan_gb300 import extensions, ics, lib
from tupan_gb300.particles import Bodies

pytestmark = pytest.mark.gpu


def particles(n, seed, prec):
    ps = ics.plummer(n, eps=1e-2, seed=seed)
    return {k: v.astype(prec) for k, v in ps.items()}


@pytest.mark.parametrize("prec", ["float64", "float32"])
def test_sizes_around_the_limit(prec):
    js = particles(5, 41, prec)
    jps = Bodies(js, dtype=np.dtype(prec))
    calc = extensions.AccJerk("CUDA", prec).calc
    old = lib.set_mode(lib.MODE_EXACT)
    try:
        for n in (1, 600, 9300, 9361, 9362, 9400, 18720, 18760, 7):
            ps = particles(n, 42 + n, prec)
            ips = Bodies(ps, dtype=np.dtype(prec))
            got = calc(ips, jps)
            want = oracle.run("acc_jerk_kernel", ps, js, prec=prec)
            for g, w in zip(got, want):
                np.testing.assert_array_equal(g, w)
            np.testing.assert_array_equal(ips.rx, ps["rx"])
    finally:
        lib.set_mode(old)


def test_read_only_inputs_are_taken():
    ps = particles(33, 50, "float64")
    ips = Bodies(ps)
    for k in ("mass", "rx", "ry", "rz", "eps2"):
        getattr(ips, k).flags.writeable = False
    old = lib.set_mode(lib.MODE_EXACT)
    try:
        got = extensions.Phi("CUDA", "float64").calc(ips, ips)[0]
    finally:
        lib.set_mode(old)
    np.testing.assert_array_equal(got, oracle.run("phi_kernel", ps, ps)[0])
