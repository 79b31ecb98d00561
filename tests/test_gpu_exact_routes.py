"""EXACT sweeps either side of each line of the dispatch (few j, few i, many
i): the oracle's bits, and no shape far off the time of its neighbours."""

import ctypes

import numpy as np
import pytest

import oracle
from tupan_gb300 import lib

pytestmark = pytest.mark.gpu
ATTRS = ("m", "rx", "ry", "rz", "e2", "vx", "vy", "vz",
         "ax", "ay", "az", "jx", "jy", "jz")
NIN = {"phi_kernel": 5, "acc_kernel": 5, "acc_jerk_kernel": 8,
       "snap_crackle_kernel": 14, "tstep_kernel": 8, "nreg_Xkernel": 8}
NOUT = {"phi_kernel": 1, "acc_kernel": 3, "acc_jerk_kernel": 6,
        "snap_crackle_kernel": 6, "tstep_kernel": 2, "nreg_Xkernel": 7}
ETA = 1.0 / 64


def bodies(n, seed, prec):
    g = np.random.default_rng(seed)
    p = {k: g.standard_normal(n) for k in ATTRS}
    p["m"] = g.random(n) / n
    p["e2"] = g.random(n) * 1e-3
    return {k: v.astype(prec) for k, v in p.items()}


class Sweep(object):
    def __init__(self, kernel, ips, jps, prec):
        import torch
        dt = torch.float64 if prec == "float64" else torch.float32
        names = ATTRS[:NIN[kernel]]
        sets = [{k: torch.from_numpy(np.ascontiguousarray(p[k])).cuda()
                 for k in names} for p in (ips, jps)]
        ni, nj = len(ips["m"]), len(jps["m"])
        self.out = [torch.full((ni,), float("nan"), dtype=dt, device="cuda")
                    for _ in range(NOUT[kernel])]
        VP = ctypes.c_void_p
        ptr = [(VP * len(names))(*[s[k].data_ptr() for k in names])
               for s in sets]
        outs = (VP * len(self.out))(*[o.data_ptr() for o in self.out])
        scal = (ctypes.c_double * 8)(ETA)
        self.args = (lib.KERNEL_ID[kernel], lib.MODE_EXACT, ni, ptr[0], nj,
                     ptr[1], scal, 0, outs, None)
        self.keep = sets
        self.L = lib.load(prec)

    def __call__(self, sync=0):
        assert self.L.tupan_gb300_dev_sweep(*self.args, sync) == 0


def check(kernel, ni, nj, prec):
    ips, jps = bodies(ni, 1, prec), bodies(nj, 2, prec)
    s = Sweep(kernel, ips, jps, prec)
    s(1)
    scal = {"tstep_kernel": {"eta": ETA}, "nreg_Xkernel": {"dt": ETA}}
    want = oracle.run(kernel, ips, jps, scal.get(kernel), prec=prec)
    for o, w in zip(s.out, want):
        np.testing.assert_array_equal(o.cpu().numpy(), w)


DOUBLE = ([(ni, nj) for ni in (1, 304, 305, 1300) for nj in (1, 2, 3, 4)] +
          [(29999, 3), (30000, 3), (30001, 4), (305, 101), (305, 102),
           (5000, 1666), (5000, 1667), (5001, 1667)])


@pytest.mark.parametrize("kernel", sorted(NIN))
@pytest.mark.parametrize("ni,nj", DOUBLE)
def test_double(kernel, ni, nj):
    check(kernel, ni, nj, "float64")


FLOAT = ([(ni, nj) for ni in (1, 129) for nj in (1, 8, 9, 16, 17)] +
         [(20000, 33), (21000, 33), (33000, 9), (36001, 9), (36000, 9)] +
         [(many + d, 130) for many in (33000, 40000, 42000, 64000)
          for d in (-1, 0, 1)])


@pytest.mark.parametrize("kernel", sorted(NIN))
@pytest.mark.parametrize("ni,nj", FLOAT)
def test_float(kernel, ni, nj):
    check(kernel, ni, nj, "float32")


def microseconds(kernel, ni, nj, prec):
    import torch
    s = Sweep(kernel, bodies(ni, 1, prec), bodies(nj, 2, prec), prec)
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
    return min(best)


@pytest.mark.parametrize("kernel", ["phi_kernel", "tstep_kernel"])
@pytest.mark.parametrize("nj", [1, 16])
def test_few_j_do_not_take_a_block_an_i(kernel, nj):
    pytest.importorskip("torch")
    assert (microseconds(kernel, 5000, nj, "float64") <
            2.0 * microseconds(kernel, 7000, nj, "float64"))


@pytest.mark.parametrize("kernel", ["acc_kernel", "acc_jerk_kernel",
                                    "snap_crackle_kernel"])
def test_many_i_in_float_fill_the_chip(kernel):
    # 3.7 times the i: with one i a thread 2.3 to 2.5 times as long, the
    # lanes of the smaller sweep being idle in part
    pytest.importorskip("torch")
    assert (microseconds(kernel, 130000, 2048, "float32") <
            2.75 * microseconds(kernel, 35000, 2048, "float32"))
