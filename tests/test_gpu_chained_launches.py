"""Sweeps whose kernels are launched as dependents of one another: back to
back on a stream, each reading what the one before wrote, they give the bits
that they give with the device idle before every launch, and under capture."""

import numpy as np
import pytest

from tupan_gb300 import ics, lib

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

ATTRS = ("m", "rx", "ry", "rz", "e2", "vx", "vy", "vz")


class Euler:
    """Euler steps whose sweeps read positions that torch has just moved."""

    def __init__(self, ni, nj, mode):
        ps = ics.plummer(nj, eps=1e-2, seed=9)
        self.d = {k: torch.from_numpy(np.ascontiguousarray(ps[k])).cuda()
                  for k in ATTRS}
        self.out = [torch.zeros(ni, dtype=torch.float64, device="cuda")
                    for _ in range(6)]
        self.ni, self.nj, self.mode = ni, nj, mode

    def steps(self, count, sync):
        pause = torch.cuda.synchronize if sync else (lambda: None)
        ps = [self.d[k].data_ptr() for k in ATTRS]
        out = [o.data_ptr() for o in self.out]
        st = torch.cuda.current_stream().cuda_stream
        for _ in range(count):
            pause()
            lib.dev_sweep("acc_jerk_kernel", self.ni, ps, self.nj, ps, out,
                          mode=self.mode, stream=st)
            pause()
            for k, o in zip(("rx", "ry", "rz"), self.out):
                self.d[k][:self.ni] += 1e-4 * o
            pause()
            lib.dev_sweep("acc_kernel", self.ni, ps[:5], self.nj, ps[:5],
                          out[3:], mode=self.mode, stream=st)
        torch.cuda.synchronize()
        lib.check()
        return [self.d[k].cpu().numpy() for k in ("rx", "ry", "rz")] + [
            o.cpu().numpy() for o in self.out]


@pytest.mark.parametrize("ni,nj,mode", [
    (100, 100, lib.MODE_EXACT), (1500, 1500, lib.MODE_EXACT),
    (60, 3000, lib.MODE_EXACT), (500, 500, lib.MODE_SPLIT),
    (200, 20000, lib.MODE_SPLIT), (9000, 9000, lib.MODE_SPLIT),
    (46400, 46400, lib.MODE_SPLIT)])
def test_back_to_back_equals_one_at_a_time(ni, nj, mode):
    want = Euler(ni, nj, mode).steps(4, sync=True)
    got = Euler(ni, nj, mode).steps(4, sync=False)
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)
    if nj > 30000:
        return
    cap = Euler(ni, nj, mode)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        warm = Euler(ni, nj, mode)
        warm.steps(1, sync=False)             # workspaces grown
        g = torch.cuda.CUDAGraph()
        ps = [cap.d[k].data_ptr() for k in ATTRS]
        out = [o.data_ptr() for o in cap.out]
        with torch.cuda.graph(g, stream=side):
            lib.dev_sweep("acc_jerk_kernel", ni, ps, nj, ps, out, mode=mode,
                          stream=side.cuda_stream)
    g.replay()
    torch.cuda.synchronize()
    one = Euler(ni, nj, mode)
    lib.dev_sweep("acc_jerk_kernel", ni, [one.d[k].data_ptr() for k in ATTRS],
                  nj, [one.d[k].data_ptr() for k in ATTRS],
                  [o.data_ptr() for o in one.out], mode=mode)
    torch.cuda.synchronize()
    lib.check()
    for a, b in zip(cap.out, one.out):
        np.testing.assert_array_equal(a.cpu().numpy(), b.cpu().numpy())
