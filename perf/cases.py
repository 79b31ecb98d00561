"""Performance cases of the kernel layer: what its users have it do.

Three ways in, as users take them: the extension objects on host arrays
(``extensions.AccJerk("CUDA", prec).calc(ps, ps)``, the drop-in interface
tupan's integrators call), ``lib.dev_sweep`` on arrays that stay in HBM, and
the device-resident integrators (a whole call: create, evolve, read the
state back).  Each kind appears in the modes it is used in: EXACT (the
default: bit-identical to tupan's C kernels) in float64 and float32, and
SPLIT (FP32 pairs on double-single positions).
"""

import math

import numpy as np
import torch

from tupan_gb300 import extensions, lib
from tupan_gb300.ensemble import DeviceEnsemble
from tupan_gb300.integrator import DeviceBlockHermite, DeviceHermite
from tupan_gb300.kepler import DeviceSakura
from tupan_gb300.particles import Bodies

ETA = 1.0 / 64
STATE = ("rx", "ry", "rz", "vx", "vy", "vz")
CLASSES = {"phi": extensions.Phi, "acc": extensions.Acc,
           "acc_jerk": extensions.AccJerk, "tstep": extensions.Tstep,
           "snap_crackle": extensions.SnapCrackle}
# flops of one interaction, as the reference counts them (tstep: no figure
# there; its operations, one per arithmetic operator)
FLOPS = {"phi": 14, "acc": 20, "acc_jerk": 42, "snap_crackle": 114,
         "tstep": 42}
N_IN = {"phi": 5, "acc": 5, "acc_jerk": 8, "snap_crackle": 14, "tstep": 8}
N_OUT = {"phi": 1, "acc": 3, "acc_jerk": 6, "snap_crackle": 6, "tstep": 2}
# attributes of dev_sweep's pointer lists, in call order
ATTRS = ("m", "rx", "ry", "rz", "e2", "vx", "vy", "vz",
         "ax", "ay", "az", "jx", "jy", "jz")


def listed():
    return [
        # one force evaluation of the CPU-runnable configuration (256-body
        # Plummer sphere) from tupan's Python integrators: latency counts
        {"name": "plugin_exact_n256", "kind": "plugin", "kernels": "acc_jerk",
         "prec": "float64", "mode": "exact", "n": 256, "eps": 1e-2},
        # the sweeps of one shared sixth-order Hermite step, odd size
        {"name": "plugin_exact_step6_n3001", "kind": "plugin",
         "kernels": "tstep,acc_jerk,snap_crackle", "prec": "float64",
         "mode": "exact", "n": 3001, "eps": 1e-3},
        # single precision runs (tupan --use_sp): energies and forces
        {"name": "plugin_exact_f32_n10007", "kind": "plugin",
         "kernels": "phi,acc", "prec": "float32", "mode": "exact",
         "n": 10007, "eps": 1e-2},
        # a large model in the default mode: energies and forces
        {"name": "plugin_exact_n32768", "kind": "plugin",
         "kernels": "phi,acc_jerk", "prec": "float64", "mode": "exact",
         "n": 32768, "eps": 1e-4},
        # smallest size of the SPLIT force-sweep configuration, with the
        # time-step sweep of a shared adaptive step
        {"name": "plugin_split_n16384", "kind": "plugin",
         "kernels": "acc_jerk,tstep", "prec": "float64", "mode": "split",
         "n": 16384, "eps": 1e-4},
        # the benchmark's step: Acc and AccJerk of 2^18 bodies, SPLIT
        {"name": "plugin_split_n262144", "kind": "plugin",
         "kernels": "acc,acc_jerk", "prec": "float64", "mode": "split",
         "n": 262144, "eps": 1e-4},
        # an active subset against all bodies on resident arrays: the
        # sweeps of one block time step of order 6
        {"name": "device_split_active_1021_65536", "kind": "device",
         "kernels": "acc_jerk,snap_crackle,tstep", "mode": "split",
         "ni": 1021, "nj": 65536, "eps": 1e-4},
        # the same in the default mode on a smaller model
        {"name": "device_exact_active_100_8192", "kind": "device",
         "kernels": "acc_jerk,tstep", "mode": "exact", "ni": 100,
         "nj": 8192, "eps": 1e-4},
        # the 256-body configuration integrated on the device, bit-identical
        # to tupan's ahermite4
        {"name": "hermite4_exact_n256", "kind": "hermite", "order": 4,
         "mode": "exact", "n": 256, "steps": 48, "eps": 1e-2},
        # individual block steps, Salpeter masses
        {"name": "block6_split_n16384", "kind": "block", "order": 6,
         "mode": "split", "n": 16384, "steps": 32, "eps": 1e-4},
        # many small systems of 3 to 512 bodies, each with its own step
        {"name": "ensemble_256", "kind": "ensemble", "systems": 256,
         "lo": 3, "hi": 512, "t_end": 1.0 / 1024, "eps": 1e-4},
        # Sakura integrator, unsoftened Salpeter sphere
        {"name": "sakura_exact_n4096", "kind": "sakura", "mode": "exact",
         "n": 4096, "steps": 2, "tau": 1.0 / 256},
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges."""
    kind = rng.choice(["plugin_exact"] * 4 + ["plugin_f32"] +
                      ["plugin_split"] * 3 + ["device_split"] +
                      ["device_exact", "hermite", "block", "ensemble",
                       "sakura"])
    eps = rng.choice([0.0, 1e-4, 1e-3, 1e-2])
    if kind == "plugin_exact":
        n = _log_size(rng, 16, 24576)
        few = ["phi", "acc", "acc_jerk", "phi,acc_jerk", "acc_jerk,tstep"]
        all6 = few + ["tstep,acc_jerk,snap_crackle"]
        return {"kind": "plugin", "kernels": rng.choice(all6 if n < 16384
                                                        else few),
                "prec": "float64", "mode": "exact", "n": n, "eps": eps}
    if kind == "plugin_f32":
        return {"kind": "plugin",
                "kernels": rng.choice(["phi", "acc", "phi,acc", "acc_jerk"]),
                "prec": "float32", "mode": "exact",
                "n": _log_size(rng, 64, 32768), "eps": max(eps, 1e-3)}
    if kind == "plugin_split":
        return {"kind": "plugin",
                "kernels": rng.choice(["phi", "acc", "acc_jerk",
                                       "acc,acc_jerk", "acc_jerk,tstep",
                                       "tstep,acc_jerk,snap_crackle"]),
                "prec": "float64", "mode": "split",
                "n": _log_size(rng, 1024, 131072), "eps": max(eps, 1e-4)}
    if kind == "device_split":
        return {"kind": "device", "kernels": "acc_jerk,snap_crackle,tstep",
                "mode": "split", "ni": _log_size(rng, 1, 16384),
                "nj": _log_size(rng, 16384, 65536), "eps": 1e-4}
    if kind == "device_exact":
        return {"kind": "device", "kernels": "acc_jerk,tstep",
                "mode": "exact", "ni": _log_size(rng, 1, 2048),
                "nj": _log_size(rng, 2048, 16384), "eps": eps}
    if kind == "hermite":
        order = rng.choice([2, 4, 6, 8])
        return {"kind": "hermite", "order": order, "mode": "exact",
                "n": _log_size(rng, 16, 384),
                "steps": 48 if order < 6 else 16, "eps": max(eps, 1e-3)}
    if kind == "block":
        return {"kind": "block", "order": rng.choice([4, 6]),
                "mode": "split", "n": _log_size(rng, 2048, 16384),
                "steps": 32, "eps": 1e-4}
    if kind == "ensemble":
        return {"kind": "ensemble", "systems": _log_size(rng, 16, 256),
                "lo": 3, "hi": rng.choice([64, 200, 512]),
                "t_end": 1.0 / 1024, "eps": 1e-4}
    return {"kind": "sakura", "mode": "exact", "n": _log_size(rng, 256, 4096),
            "steps": 2, "tau": 1.0 / 256}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _sphere(n, eps, rng, salpeter=False):
    """A Plummer sphere in N-body units (G = M = 1, E = -1/4), e2 =
    eps^2/2 per body; ax .. jz hold the sphere's mean-field acceleration and
    jerk, what a predictor hands to the snap/crackle sweep."""
    if salpeter:                     # dN/dm ~ m^-2.35 on [0.1, 100]
        lo, hi = 0.1 ** -1.35, 100.0 ** -1.35
        m = (lo + rng.random(n) * (hi - lo)) ** (-1.0 / 1.35)
        m /= m.sum()
    else:
        m = np.full(n, 1.0 / n)
    x = (rng.permutation(n) + rng.random(n)) * 0.999 / n
    r = 1.0 / np.sqrt(x ** (-2.0 / 3.0) - 1.0)
    q = np.empty(n)
    todo = np.arange(n)
    while todo.size:
        a, b = rng.random(todo.size), rng.random(todo.size) * 0.1
        ok = b < a * a * (1.0 - a * a) ** 3.5
        q[todo[ok]] = a[ok]
        todo = todo[~ok]
    speed = q * math.sqrt(2.0) * (1.0 + r * r) ** -0.25

    def directed(length):
        c = rng.uniform(-1.0, 1.0, n)
        p = rng.uniform(0.0, 2.0 * math.pi, n)
        s = np.sqrt(1.0 - c * c)
        v = np.stack([length * s * np.cos(p), length * s * np.sin(p),
                      length * c])
        return v - (v * m).sum(axis=1, keepdims=True)

    scale = 3.0 * math.pi / 16.0
    pos = directed(r) * scale
    vel = directed(speed) / math.sqrt(scale)
    d2 = (pos * pos).sum(axis=0) + scale * scale
    rv = (pos * vel).sum(axis=0)
    acc = -pos * d2 ** -1.5
    jrk = -(vel - 3.0 * (rv / d2) * pos) * d2 ** -1.5
    out = {"m": m, "e2": np.full(n, eps * eps / 2.0)}
    for k, vec in (("r", pos), ("v", vel), ("a", acc), ("j", jrk)):
        for c in range(3):
            out[k + "xyz"[c]] = np.ascontiguousarray(vec[c])
    return out


def _inputs(case, seed):
    """Host arrays of the case (a list of systems for an ensemble, an (i, j)
    pair of sets for resident arrays)."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "ensemble":
        # sizes spread evenly over [lo, hi], the same for every seed
        span = case["hi"] - case["lo"] + 1
        sizes = [case["lo"] + int(span * math.fmod((k + 0.5) * 0.618033988749,
                                                   1.0))
                 for k in range(case["systems"])]
        return [_sphere(n, case["eps"], rng) for n in sizes]
    if kind == "sakura":
        return _sphere(case["n"], 0.0, rng, salpeter=True)
    if kind == "block":
        return _sphere(case["n"], case["eps"], rng, salpeter=True)
    if kind == "device":
        j = _sphere(case["nj"], case["eps"], rng)
        pick = np.sort(rng.permutation(case["nj"])[:case["ni"]])
        return {k: np.ascontiguousarray(v[pick]) for k, v in j.items()}, j
    ps = _sphere(case["n"], case["eps"], rng)
    if kind == "plugin" and case["prec"] == "float32":
        ps = {k: v.astype(np.float32) for k, v in ps.items()}
    return ps


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    src = _inputs(case, seed)
    if kind == "plugin":
        st["ext"] = [(k, CLASSES[k]("CUDA", case["prec"]))
                     for k in case["kernels"].split(",")]
        st["ps"] = Bodies(src, dtype=np.dtype(case["prec"]))
        st["mode"] = lib.MODE_SPLIT if case["mode"] == "split" \
            else lib.MODE_EXACT
    elif kind == "device":
        lib.load("float64")
        ips, jps = ({k: torch.from_numpy(v).cuda() for k, v in s.items()}
                    for s in src)
        st["i"], st["j"], st["out"] = ips, jps, {}
        for k in case["kernels"].split(","):
            st["out"][k] = [torch.empty(case["ni"], dtype=torch.float64,
                                        device="cuda")
                            for _ in range(N_OUT[k])]
        torch.cuda.synchronize()
    else:
        lib.load("float64")
        st["systems"] = src
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "plugin":
        if case["prec"] == "float64":
            lib.set_mode(st["mode"])
        ps, out = st["ps"], []
        for k, ext in st["ext"]:
            out.extend(ext.calc(ps, ps, *((ETA,) if k == "tstep" else ())))
        return out
    if kind == "device":
        out = []
        for k, dst in st["out"].items():
            names = ATTRS[:N_IN[k]]
            lib.dev_sweep(k + "_kernel", case["ni"],
                          [st["i"][a].data_ptr() for a in names], case["nj"],
                          [st["j"][a].data_ptr() for a in names],
                          [o.data_ptr() for o in dst], scal=[ETA],
                          mode=lib.MODE_SPLIT if case["mode"] == "split"
                          else lib.MODE_EXACT)
            out.extend(dst)
        return out
    if kind == "hermite":
        d = DeviceHermite(st["systems"], ETA, order=case["order"],
                          mode=case["mode"])
        t = d.evolve(1e3, max_steps=case["steps"])
        s = d.state()
        steps = d.nsteps
        d.close()
        return [s[k] for k in STATE] + [t, steps]
    if kind == "block":
        d = DeviceBlockHermite(st["systems"], 2 * ETA, 1.0 / 32,
                               order=case["order"], mode=case["mode"])
        t = d.evolve(1e3, max_steps=case["steps"])
        s = d.state()
        act = d.active
        d.close()
        return [s[k] for k in STATE] + [s["t"], s["dt"], t, act]
    if kind == "ensemble":
        d = DeviceEnsemble(st["systems"], ETA)
        d.evolve(case["t_end"])
        t, steps, s = d.state()
        d.close()
        return [s[k] for k in STATE] + [t, steps]
    d = DeviceSakura(st["systems"], mode=case["mode"])
    t, steps, _ = d.evolve(case["tau"], case["tau"] * case["steps"])
    s = d.state()
    d.close()
    return [s[k] for k in STATE] + [t, steps]


def work(case):
    """Bytes: each particle attribute read once and each result written
    once; flops: the reference's count per interaction."""
    kind = case["kind"]
    if kind in ("plugin", "device"):
        ni = case.get("ni", case.get("n"))
        nj = case.get("nj", ni)
        size = 4 if case.get("prec") == "float32" else 8
        ks = case["kernels"].split(",")
        sets = nj if kind == "plugin" else ni + nj
        return {"bytes": size * (max(N_IN[k] for k in ks) * sets +
                                 sum(N_OUT[k] for k in ks) * ni),
                "flops": sum(FLOPS[k] for k in ks) * ni * nj}
    if kind == "ensemble":
        mean = 0.5 * (case["lo"] + case["hi"])
        n2 = (case["lo"] ** 2 + case["lo"] * case["hi"] +
              case["hi"] ** 2) / 3.0
        steps = 24      # a typical system's steps to t_end
        return {"bytes": 8 * 14 * mean * case["systems"],
                "flops": (FLOPS["tstep"] + 3 * FLOPS["acc_jerk"]) * n2 *
                case["systems"] * steps}
    n, steps = case["n"], case["steps"]
    if kind == "sakura":
        # two sweeps a step, about 60 operations a leapfrog pair
        return {"bytes": 8 * 14 * n, "flops": 2 * 60 * steps * n * n}
    if kind == "hermite":
        f = {2: FLOPS["acc"], 4: FLOPS["acc_jerk"]}.get(
            case["order"], FLOPS["acc_jerk"] + FLOPS["snap_crackle"])
        return {"bytes": 8 * 14 * n,
                "flops": (FLOPS["tstep"] + 3 * f) * steps * n * n}
    f = FLOPS["acc_jerk"] + (FLOPS["snap_crackle"] if case["order"] > 4
                             else 0)
    # the start's full sweeps, then about a sixteenth active a step
    return {"bytes": 8 * 16 * n,
            "flops": (f + FLOPS["tstep"]) * n * n +
            (2 * f + FLOPS["tstep"]) * steps * n * n / 16}


# ---------------------------------------------------------------------------
# The same results in 64 bits from torch
# ---------------------------------------------------------------------------
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t64(src):
    return {k: torch.from_numpy(np.asarray(v, dtype=np.float64)).to(_dev())
            for k, v in src.items()}


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _pair_terms(kernels, I, J):
    """Per-kernel outputs of the i rows I against all of J: tensors [..., ni],
    [..., nj]; sums over the last axis."""
    def diff(q):
        return [I[q + c].unsqueeze(-1) - J[q + c].unsqueeze(-2)
                for c in "xyz"]

    res = {}
    d = diff("r")
    r2 = _dot(d, d)
    q = torch.where(r2 > 0, 1.0 / (r2 + (I["e2"].unsqueeze(-1) +
                                         J["e2"].unsqueeze(-2))), 0.0)
    mj = J["m"].unsqueeze(-2)
    k1 = q.sqrt()
    if "phi" in kernels:
        res["phi"] = [-(mj * k1).sum(-1)]
    k3 = mj * q * k1
    if "acc" in kernels or "acc_jerk" in kernels:
        acc = [-(k3 * x).sum(-1) for x in d]
        if "acc" in kernels:
            res["acc"] = acc
    if not {"acc_jerk", "snap_crackle", "tstep"} & set(kernels):
        return res
    u = diff("v")
    rv = _dot(d, u)
    if "acc_jerk" in kernels:
        al = 3.0 * rv * q
        res["acc_jerk"] = acc + [-(k3 * (y - al * x)).sum(-1)
                                 for x, y in zip(d, u)]
    if "tstep" in kernels:
        ms = I["m"].unsqueeze(-1) + mj
        phi = ms * k1
        w2 = q * (_dot(u, u) + 2.0 * phi)
        g = q * (w2 + 2.0 * q * phi) * (ETA * _tstep_scale(I) / w2.sqrt())
        w2 = torch.where(r2 > 0, w2 - g * rv, 0.0)
        e = ETA * _tstep_scale(I)
        res["tstep"] = [e / (1.0 + w2.sum(-1)).sqrt(),
                        e / (1.0 + w2.amax(-1).clamp_min(0.0)).sqrt()]
    if "snap_crackle" in kernels:
        a, j = diff("a"), diff("j")
        al = rv * q
        be = 3.0 * ((_dot(u, u) + _dot(d, a)) * q + al * al)
        ga = (3.0 * _dot(u, a) + _dot(d, j)) * q + al * (be - 4.0 * al * al)
        u1 = [y - 3.0 * al * x for x, y in zip(d, u)]
        a1 = [z - 6.0 * al * y - be * x for x, y, z in zip(d, u1, a)]
        j1 = [w - 9.0 * al * z - 3.0 * be * y - 3.0 * ga * x
              for x, y, z, w in zip(d, u1, a1, j)]
        res["snap_crackle"] = [-(k3 * x).sum(-1) for x in a1 + j1]
    return res


def _tstep_scale(I):
    return I.get("eta_scale", 1.0)


def _sweeps(kernels, I, J):
    """The kernels' outputs, i rows taken in chunks that fit the card."""
    ni, nj = I["m"].shape[-1], J["m"].shape[-1]
    rows = max(1, (1 << 24) // nj)
    parts = {k: [] for k in kernels}
    for lo in range(0, ni, rows):
        sub = {k: (v[lo:lo + rows] if torch.is_tensor(v) else v)
               for k, v in I.items()}
        for k, v in _pair_terms(kernels, sub, J).items():
            parts[k].append(v)
    return {k: [torch.cat([p[c] for p in v]) for c in range(N_OUT[k])]
            for k, v in parts.items()}


def _add_forces(ps, kernels, I=None):
    """acc/jerk (then snap/crackle with those) of I against ps, as a dict."""
    I = ps if I is None else I
    f = {}
    for k, names in (("acc", "a"), ("acc_jerk", "aj"), ("snap_crackle", "sc")):
        if k in kernels:
            J = ps if I is not ps else dict(ps, **f)
            out = _sweeps([k], dict(I, **f), J)[k]
            f.update({a + c: out[3 * p + q] for p, a in enumerate(names)
                      for q, c in enumerate("xyz")})
    return f


def _predict(order, s, f, h, c):
    """Taylor increments of r and v of component c over h."""
    d = [s["v" + c]] + [f[k + c] for k in {2: "a", 4: "aj", 6: "ajs",
                                           8: "ajsc"}[order]]
    r = v = 0.0
    for k in range(len(d) - 1, -1, -1):
        r = (r + d[k]) * h / (k + 1)
        if k:
            v = (v + d[k]) * h / k
    return r, v


def _corrector(order, s0, f0, f1, h, c):
    """Hermite corrector of component c: new r, v from both ends."""
    def integral(x0, lower, upper):
        p = [(lower[k], upper[k]) for k in range(len(lower))]
        a = p[0][0] + p[0][1]
        if order == 2:
            return x0 + a * h / 2
        b = p[1][0] - p[1][1]
        if order == 4:
            return x0 + (b * h / 6 + a) * h / 2
        s = p[2][0] + p[2][1]
        if order == 6:
            return x0 + ((s * h / 12 + b) * h / 5 + a) * h / 2
        e = p[3][0] - p[3][1]
        return x0 + (((e * h / 20 + s) * h / 3 + 3 * b) * h / 14 + a) * h / 2

    names = {2: "a", 4: "aj", 6: "ajs", 8: "ajsc"}[order]
    lo = [f0[k + c] for k in names]
    up = [f1[k + c] for k in names]
    v1 = integral(s0["v" + c], lo, up)
    r1 = integral(s0["r" + c], [s0["v" + c]] + lo[:-1], [v1] + up[:-1])
    return r1, v1


def _force_kernels(order):
    return {2: ["acc"], 4: ["acc_jerk"]}.get(order,
                                             ["acc_jerk", "snap_crackle"])


def _quantised(dt, t, cap):
    """tupan's power-of-two step for a least pair step dt at time t."""
    b = 2.0 ** int(math.log2(dt) - 1)
    while math.fmod(t + b, b) != 0:
        b /= 2
    return min(b, cap)


def _exact_hermite(case, seed):
    ps = _t64(_inputs(case, seed))
    order, ks, t = case["order"], _force_kernels(case["order"]), 0.0
    for _ in range(case["steps"]):
        dt = _sweeps(["tstep"], ps, ps)["tstep"][0].abs().min().item()
        h = _quantised(dt, t, ETA)
        p0 = dict(ps)
        f0 = _add_forces(p0, ks)
        for c in "xyz":
            r, v = _predict(order, p0, f0, h, c)
            ps["r" + c], ps["v" + c] = p0["r" + c] + r, p0["v" + c] + v
        for _ in range(2):
            f1 = _add_forces(ps, ks)
            new = [_corrector(order, p0, f0, f1, h, c) for c in "xyz"]
            for c, (r, v) in zip("xyz", new):
                ps["r" + c], ps["v" + c] = r, v
        t += h
    return [ps[k] for k in STATE] + [t, case["steps"]]


def _exact_block(case, seed):
    order, eta, cap = case["order"], 2 * ETA, 1.0 / 32
    ks = _force_kernels(order)
    s = _t64({k: v for k, v in _inputs(case, seed).items() if k[0] in "mer"
              or k[0] == "v"})
    der = "aj" if order == 4 else "ajsc"
    s.update(_add_forces(s, ks))
    tn = torch.zeros_like(s["m"])
    scale = {"eta_scale": eta / ETA}

    def steps_of(I, J, t):
        dts = _sweeps(["tstep"], dict(I, **scale), J)["tstep"][0].abs()
        return torch.tensor([_quantised(x, t, cap) for x in dts.tolist()],
                            dtype=torch.float64, device=tn.device)

    dt = steps_of(s, s, 0.0)
    t, active = 0.0, 0
    for _ in range(case["steps"]):
        t = (tn + dt).min().item()
        act = torch.nonzero(tn + dt == t).squeeze(1)
        active += int(act.numel())
        h = t - tn
        J = {"m": s["m"], "e2": s["e2"]}
        for c in "xyz":                  # r, v, a, j at the block time
            chain = [s[k + c] for k in "rv" + der]
            for p, k in enumerate("rvaj"):
                x = chain[-1] if p < len(chain) else 0.0
                for q in range(len(chain) - 2, p - 1, -1):
                    x = chain[q] + h * x / (q - p + 1)
                J[k + c] = x
        i0 = {k: v[act] for k, v in s.items()}
        hi = dt[act]
        for _ in range(2):
            I = {k: v[act] for k, v in J.items()}
            f1 = _add_forces(J, ks, I)
            new = {}
            for c in "xyz":
                new["r" + c], new["v" + c] = _corrector(order, i0, i0, f1,
                                                        hi, c)
            new.update({k: v for k, v in f1.items() if k[0] in "aj"})
            for k, v in new.items():
                J[k] = J[k].clone()
                J[k][act] = v
        for k in STATE:
            s[k] = s[k].clone()
            s[k][act] = J[k][act]
        for k, v in f1.items():
            s[k] = s[k].clone()
            s[k][act] = v
        dt[act] = steps_of({k: v[act] for k, v in J.items()}, J, t)
        tn[act] = t
    return [s[k] for k in STATE] + [tn, dt, t, active]


def _exact_ensemble(case, seed):
    systems = _inputs(case, seed)
    width = max(len(p["m"]) for p in systems)
    ps = {}
    for k in ("m", "e2") + STATE:
        a = np.zeros((len(systems), width))
        for row, p in enumerate(systems):
            a[row, :len(p["m"])] = p[k]
            if k == "rx":            # massless bodies out of everyone's way
                a[row, len(p["m"]):] = 1e6 * (2 + np.arange(
                    width - len(p["m"])))
        ps[k] = torch.from_numpy(a).to(_dev())
    real = torch.zeros_like(ps["m"], dtype=torch.bool)
    for row, p in enumerate(systems):
        real[row, :len(p["m"])] = True
    t = [0.0] * len(systems)
    steps = [0] * len(systems)
    t_end = case["t_end"]
    while min(t) < t_end:
        live = [k for k in range(len(systems)) if t[k] < t_end]
        s0 = {k: v[live] for k, v in ps.items()}
        dts = _pair_terms(["tstep"], s0, s0)["tstep"][0].abs()
        dts = torch.where(real[live], dts, math.inf).amin(-1).tolist()
        hs = []
        for k, x in zip(live, dts):
            cap = max(min(t_end - t[k], ETA), t_end * 2.0 ** -51)
            hs.append(_quantised(x, t[k], cap))
        h = torch.tensor(hs, dtype=torch.float64, device=_dev()).unsqueeze(1)
        names = [a + c for a in "aj" for c in "xyz"]

        def force(s):
            return dict(zip(names, _pair_terms(["acc_jerk"], s,
                                               s)["acc_jerk"]))

        f0 = force(s0)
        s = dict(s0)
        for c in "xyz":
            r, v = _predict(4, s0, f0, h, c)
            s["r" + c], s["v" + c] = s0["r" + c] + r, s0["v" + c] + v
        for _ in range(2):
            f1 = force(s)
            new = [_corrector(4, s0, f0, f1, h, c) for c in "xyz"]
            for c, (r, v) in zip("xyz", new):
                s["r" + c], s["v" + c] = r, v
        for k in STATE:
            ps[k][live] = s[k]
        for k, x in zip(live, hs):
            t[k] += x
            steps[k] += 1
    flat = [ps[k][real] for k in STATE]
    return flat + [np.array(t), np.array(steps, np.int64)]


def _stumpff(z):
    """c1, c2, c3 of z (positive: elliptic): sin(w)/w, (1-cos w)/z,
    (w - sin w)/w^3 with w = sqrt z; series near zero."""
    w = z.abs().sqrt().clamp_min(1e-300)
    ell = z > 0
    sn = torch.where(ell, w.sin(), w.clamp_max(700).sinh())
    half = torch.where(ell, (w / 2).sin(), (w / 2).clamp_max(350).sinh())
    c1, c2 = sn / w, 2 * (half / w) ** 2
    c3 = torch.where(ell, w - sn, sn - w) / w ** 3
    small = z.abs() < 1.0
    out = []
    for k, c in ((1, c1), (2, c2), (3, c3)):
        ser, term = torch.zeros_like(z), torch.ones_like(z) / math.factorial(k)
        for q in range(14):
            ser = ser + term
            term = -term * z / ((2 * q + k + 1) * (2 * q + k + 2))
        out.append(torch.where(small, ser, c))
    return out


def _kepler(dt, m, p, v):
    """Two-body motion over dt in universal variables, Laguerre-Conway
    iteration (lists of three tensors in, the same out)."""
    r0 = _dot(p, p).sqrt()
    eta = _dot(p, v)
    al = 2 * m / r0 - _dot(v, v)
    s = dt / r0
    for _ in range(40):
        c1, c2, c3 = _stumpff(al * s * s)
        f = r0 * s * c1 + eta * s * s * c2 + m * s ** 3 * c3 - dt
        c0 = 1 - al * s * s * c2
        f1 = r0 * c0 + eta * s * c1 + m * s * s * c2
        f2 = (m - al * r0) * s * c1 + eta * c0
        root = (16 * f1 * f1 - 20 * f * f2).abs().sqrt()
        s = s - 5 * f / (f1 + torch.where(f1 > 0, root, -root))
    c1, c2, c3 = _stumpff(al * s * s)
    g2, g3 = s * s * c2, s ** 3 * c3
    rn = r0 * (1 - al * g2) + eta * s * c1 + m * g2
    lf, lg = 1 - m * g2 / r0, dt - m * g3
    ld, le = -m * s * c1 / (r0 * rn), 1 - m * g2 / rn
    return ([lf * x + lg * y for x, y in zip(p, v)],
            [ld * x + le * y for x, y in zip(p, v)])


def _sakura_increments(ps, dt, flag):
    """sum_j (m_j / M) (two-body step with the drift taken out) of every i."""
    n = ps["m"].shape[0]
    rows = max(1, (1 << 23) // n)
    parts = []
    for lo in range(0, n, rows):
        I = {k: v[lo:lo + rows] for k, v in ps.items()}
        p0 = [I["r" + c].unsqueeze(1) - ps["r" + c] for c in "xyz"]
        v0 = [I["v" + c].unsqueeze(1) - ps["v" + c] for c in "xyz"]
        m = I["m"].unsqueeze(1) + ps["m"]
        p = [x - y * dt for x, y in zip(p0, v0)] if flag < 0 else p0
        # far pairs: one kick at the midpoint
        half = [x + y * (dt / 2) for x, y in zip(p, v0)]
        h2 = _dot(half, half)
        k = torch.where(h2 > 0, m * h2 ** -1.5, 0.0)
        v1 = [y - k * x * dt for x, y in zip(half, v0)]
        p1 = [x + y * (dt / 2) for x, y in zip(half, v1)]
        # close pairs: the Kepler solution
        bound = 64 * m / _dot(v0, v0)
        r2 = _dot(p, p)
        near = (r2 <= bound * bound) & (r2 > 0)
        b, e = _kepler(dt, m[near], [x[near] for x in p],
                       [y[near] for y in v0])
        for c in range(3):
            p1[c][near] = b[c]
            v1[c][near] = e[c]
            same = r2 == 0
            p1[c][same], v1[c][same] = p0[c][same], v0[c][same]
        if flag > 0:
            p1 = [x - y * dt for x, y in zip(p1, v1)]
        mu = ps["m"] / m
        parts.append([(mu * (a - b)).sum(1) for a, b in
                      zip(p1 + v1, p0 + v0)])
    return [torch.cat([q[c] for q in parts]) for c in range(6)]


def _exact_sakura(case, seed):
    ps = _t64(_inputs(case, seed))
    tau = case["tau"]
    for _ in range(case["steps"]):
        for flag in (0, -1, 1, 0):
            if flag:
                inc = _sakura_increments(ps, tau / 2, flag)
                for k, x in zip(STATE, inc):
                    ps[k] = ps[k] + x
            else:
                for c in "xyz":
                    ps["r" + c] = ps["r" + c] + ps["v" + c] * tau / 2
    return [ps[k] for k in STATE] + [tau * case["steps"], case["steps"]]


def exact(case, seed):
    kind = case["kind"]
    if kind == "hermite":
        return _exact_hermite(case, seed)
    if kind == "block":
        return _exact_block(case, seed)
    if kind == "ensemble":
        return _exact_ensemble(case, seed)
    if kind == "sakura":
        return _exact_sakura(case, seed)
    src = _inputs(case, seed)
    I, J = (_t64(s) for s in (src if kind == "device" else (src, src)))
    ks = case["kernels"].split(",")
    snap = kind == "plugin" and "snap_crackle" in ks
    res = _sweeps([k for k in ks if not (snap and k == "snap_crackle")], I, J)
    if snap:       # takes the acceleration and jerk just computed
        names = [a + c for a in "aj" for c in "xyz"]
        I.update(zip(names, res["acc_jerk"]))
        res.update(_sweeps(["snap_crackle"], I, I))
    return [x for k in ks for x in res[k]]
