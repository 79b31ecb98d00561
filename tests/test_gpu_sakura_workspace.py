"""The workspace that the queued Sakura sweep keeps between calls."""

from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from tupan_gb300 import ics, lib
from tupan_gb300 import kepler as kp

pytestmark = pytest.mark.gpu
NAMES = ("m", "rx", "ry", "rz", "e2", "vx", "vy", "vz")


def system(n, seed):
    torch = pytest.importorskip("torch")
    ps = ics.plummer(n, eps=0.0, seed=seed, masses="salpeter")
    return ({k: torch.from_numpy(np.ascontiguousarray(ps[k])).cuda()
             for k in NAMES},
            [torch.zeros(n, dtype=torch.float64, device="cuda")
             for _ in range(6)])


def sweep(d, out, n, mode="exact", stream=None):
    ptr = [d[k].data_ptr() for k in NAMES]
    return kp.sakura_queue(n, ptr, n, ptr, [o.data_ptr() for o in out],
                           1.0 / 512, -1, mode=mode, stream=stream)[0]


@pytest.mark.parametrize("mode", ["exact", "split"])
def test_a_sweep_after_one_too_large_for_the_memory(mode):
    n = 257
    d, out = system(n, 21)
    nk = sweep(d, out, n, mode)
    want = [o.cpu().numpy() for o in out]
    # counts of 2^40 particles (4 TiB) cannot be had: refused before any
    # launch or access
    ptr = [d[k].data_ptr() for k in NAMES]
    with pytest.raises(lib.TupanGB300Error, match="status 1"):
        kp.sakura_queue(1 << 40, ptr, 1, ptr, [o.data_ptr() for o in out],
                        1.0 / 512, -1, mode=mode)
    for m in (n, 2 * n):            # the counts fit the old size; grow again
        d, out = system(m, 21)
        for o in out:
            o.fill_(float("nan"))
        got = sweep(d, out, m, mode)
        if m == n:
            assert got == nk
            for o, w in zip(out, want):
                np.testing.assert_array_equal(o.cpu().numpy(), w)
        else:
            assert all(np.isfinite(o.cpu().numpy()).all() for o in out)


def test_systems_stepped_from_several_threads():
    # sizes apart, so that the workspace grows under way; every system's bits
    # are those of stepping it alone
    sizes = (180, 700, 1201, 333)

    def step(n, seed):
        dev = kp.DeviceSakura(ics.plummer(n, eps=0.0, seed=seed,
                                          masses="salpeter"))
        got = []
        for k in range(1, 9):
            dev.evolve(1.0 / 256, k / 256.0)
            got.append(dev.state())
        dev.close()
        return got

    want = [step(n, n) for n in sizes]
    with ThreadPoolExecutor(len(sizes)) as pool:
        runs = [pool.submit(step, n, n) for n in sizes for _ in range(2)]
        for k, r in enumerate(runs):
            for a, b in zip(r.result(), want[k // 2]):
                for c in a:
                    np.testing.assert_array_equal(a[c], b[c])


def test_sweeps_and_pair_solves_on_streams_of_several_threads():
    torch = pytest.importorskip("torch")
    sizes = (150, 900, 64, 2001)
    sys_ = [system(n, n) for n in sizes]
    rng = np.random.default_rng(3)
    m = torch.from_numpy(rng.uniform(1e-4, 1e-2, 500)).cuda()
    e2 = torch.zeros(500, dtype=torch.float64, device="cuda")
    st = torch.from_numpy(rng.standard_normal((500, 6)) * 0.05).cuda()

    def pairs(stream):
        out = torch.zeros((500, 6), dtype=torch.float64, device="cuda")
        torch.cuda.current_stream().synchronize()
        kp.kepler_pairs(500, 1.0 / 512, m, e2, st, out, stream=stream)
        return out.cpu().numpy()

    want = []
    for (d, out), n in zip(sys_, sizes):
        for mode in ("exact", "split"):
            nk = sweep(d, out, n, mode)
            want.append((nk, [o.cpu().numpy() for o in out]))
    want_pairs = pairs(None)
    torch.cuda.synchronize()

    def work(k):
        (d, out), n = sys_[k], sizes[k]
        s = torch.cuda.Stream()
        for _ in range(6):
            for q, mode in enumerate(("exact", "split")):
                nk = sweep(d, out, n, mode, s.cuda_stream)
                w = want[2 * k + q]
                assert nk == w[0]
                for o, x in zip(out, w[1]):
                    np.testing.assert_array_equal(o.cpu().numpy(), x)
            np.testing.assert_array_equal(pairs(s.cuda_stream), want_pairs)

    with ThreadPoolExecutor(len(sizes)) as pool:
        list(pool.map(work, range(len(sizes))))
