"""The two forms of the grid j-split reduction: an i's sums have the same bits
either side of the line between them, and few splits of many i cost little."""

import ctypes

import numpy as np
import pytest

from tupan_gb300 import lib

pytestmark = pytest.mark.gpu
ATTRS = ("m", "rx", "ry", "rz", "e2", "vx", "vy", "vz",
         "ax", "ay", "az", "jx", "jy", "jz")
NIN = {"phi_kernel": 5, "acc_kernel": 5, "acc_jerk_kernel": 8,
       "snap_crackle_kernel": 14, "tstep_kernel": 8, "pnacc_kernel": 8}
NOUT = {"phi_kernel": 1, "acc_kernel": 3, "acc_jerk_kernel": 6,
        "snap_crackle_kernel": 6, "tstep_kernel": 2, "pnacc_kernel": 3}


def bodies(n, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    p = {k: torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
         for k in ATTRS}
    p["m"] = p["m"].abs() / n
    p["e2"].fill_(1e-4)
    return p


class Sweep(object):
    def __init__(self, kernel, ni, ips, nj, jps):
        import torch
        names = ATTRS[:NIN[kernel]]
        self.out = [torch.full((ni,), float("nan"), dtype=torch.float64,
                               device="cuda") for _ in range(NOUT[kernel])]
        VP = ctypes.c_void_p
        ptr = [(VP * len(names))(*[s[k].data_ptr() for k in names])
               for s in (ips, jps)]
        scal = (ctypes.c_double * 8)(1.0 / 64, *[0.01 ** k
                                                 for k in range(1, 8)])
        outs = (VP * len(self.out))(*[o.data_ptr() for o in self.out])
        self.args = (lib.KERNEL_ID[kernel], lib.MODE_SPLIT, ni, ptr[0], nj,
                     ptr[1], scal, 4, outs, None)
        self.L = lib.load()

    def __call__(self, sync=0):
        assert self.L.tupan_gb300_dev_sweep(*self.args, sync) == 0


@pytest.mark.parametrize("kernel", sorted(NIN))
@pytest.mark.parametrize("gsplit", [9, 12, 15, 16, 17, 23, 24, 25, 31, 32])
def test_same_bits_either_side_of_the_line(kernel, gsplit):
    pytest.importorskip("torch")
    n, nj = 1500 * gsplit, 256 * gsplit - 100
    ips, jps = bodies(n, 1), bodies(nj, 2)
    lib.set_centred(0)
    lib.set_split_config(kernel, 0, gsplit)
    try:
        sweeps = [Sweep(kernel, ni, ips, nj, jps) for ni in (n - 1, n)]
        for s in sweeps:
            s(1)
    finally:
        lib.set_split_config(kernel, -1, 0)
        lib.set_centred(-1)
    for a, b in zip(*[s.out for s in sweeps]):
        a, b = a.cpu().numpy(), b.cpu().numpy()
        assert np.isfinite(b).all()
        np.testing.assert_array_equal(a, b[:-1])


# one run of pairs in each split: its double sum is the sweep of those j
# alone, whose unsplit result has no reduction.  Sums and maxima (Tstep is
# left out: its last step is not linear) against adding those in order; one
# split is exact, each further addition rounds once
@pytest.mark.parametrize("kernel", ["phi_kernel", "acc_kernel",
                                    "acc_jerk_kernel", "snap_crackle_kernel",
                                    "pnacc_kernel"])
@pytest.mark.parametrize("gsplit", [2, 3, 7, 8])
def test_few_splits_add_their_parts(kernel, gsplit):
    pytest.importorskip("torch")
    ni, nj = 1300, 256 * gsplit
    ips, jps = bodies(ni, 3), bodies(nj, 4)
    lib.set_centred(0)
    try:
        lib.set_split_config(kernel, 0, gsplit)
        whole = Sweep(kernel, ni, ips, nj, jps)
        whole(1)
        lib.set_split_config(kernel, 0, 1)
        parts = []
        for y in range(gsplit):
            cut = {k: v[256 * y:256 * (y + 1)].contiguous()
                   for k, v in jps.items()}
            s = Sweep(kernel, ni, ips, 256, cut)
            s(1)
            parts.append(s.out)
    finally:
        lib.set_split_config(kernel, -1, 0)
        lib.set_centred(-1)
    for c, got in enumerate(whole.out):
        want = np.zeros(ni)
        for p in parts:
            want = want + p[c].cpu().numpy()
        np.testing.assert_array_equal(got.cpu().numpy(), want)


def microseconds(kernel, ni, nj, gsplit):
    import torch
    lib.set_centred(0)
    lib.set_split_config(kernel, 0, gsplit)
    try:
        s = Sweep(kernel, ni, bodies(ni, 1), nj, bodies(nj, 2))
        for _ in range(3):
            s()
        best = []
        for _ in range(7):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            for _ in range(10):
                s()
            b.record()
            torch.cuda.synchronize()
            best.append(a.elapsed_time(b) * 100)
    finally:
        lib.set_split_config(kernel, -1, 0)
        lib.set_centred(-1)
    return min(best)


def test_splits_of_many_i_cost_little():
    # 250000 x 2048 in one part against eight: the partial sums, 96 MB
    # written and read, against a sweep that is better balanced
    pytest.importorskip("torch")
    one, eight = (microseconds("acc_jerk_kernel", 250000, 2048, g)
                  for g in (1, 8))
    assert eight < 0.95 * one, (one, eight)
