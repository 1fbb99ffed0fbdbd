"""The workloads that the speed of this library is judged by, each through its public entry points.

They are what users of the library do: one spectrum while a protocol is being set up, batches of
voxels, isochromat spreads, fingerprint dictionaries, fits of saturation ladders and of pulsed trains,
joint fits of uneven batches, and the warm-start network. Models and sequences are those of bench.py
and of the tests (an amide pool, amide + NOE + super-Lorentzian MT, four or five pools with MT at 3 T,
the creatine phantom); voxel counts, offsets, pulses and samples spread over the ranges these meet.

  listed()   the named cases          draw(rng)  one more case of the same ranges
  prepare()  what a program holds     run()      one pass
  work()     its least work           tolerance(), exact()  what its outputs may differ by

`exact` restates the model in plain torch, float64: the generator of every event, torch.matrix_exp,
and the Levenberg-Marquardt rules, without this library's code.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "bmc-jax_b200"))

GAMMA, B0 = 267.5153, 3.0
HZ_PPM = 42.5764 * B0
# (dw ppm, T1 s, T2 s): amide, amine, hydroxyl, NOE, creatine
POOLS = [(3.5, 1.0, 0.1), (2.0, 1.0, 0.1), (1.0, 1.0, 0.1), (-3.5, 1.3, 0.005), (1.9, 1.0, 0.03)]
PRECISION = {"f64": 0, "f32": 1, "mixed": 2}


def listed():
    return [
        # the smallest call: one Z-spectrum of one tissue, continuous-wave saturation (a protocol being
        # set up, an interactive plot)
        {"name": "cw_one", "kind": "cw", "voxels": 1, "offsets": 61, "pools": 2, "mt": True, "tsat": 2.0, "b1": 1.0},
        # one tissue under the pulsed train of a scanner's sequence file: 20 shaped pulses with a running
        # phase, a spoiler and a delay of its own after each (the phantom tables of the tests)
        {"name": "train_one", "kind": "train", "style": "scanner", "precision": "f64", "voxels": 1, "offsets": 102,
         "pools": 1, "mt": False, "pulses": 20, "samples": 200, "tp": 0.1, "b1": 0.8},
        # a slice of voxels, float64: the benchmark's train (20 Gaussian pulses of 200 samples)
        {"name": "train_voxels", "kind": "train", "style": "regular", "precision": "f64", "voxels": 193, "offsets": 101,
         "pools": 4, "mt": True, "pulses": 20, "samples": 200, "tp": 0.05, "b1": 1.0},
        # the largest: a volume in mixed precision, device arrays in and out
        {"name": "train_volume", "kind": "train", "style": "regular", "precision": "mixed", "device": True,
         "voxels": 2048, "offsets": 101, "pools": 4, "mt": True, "pulses": 20, "samples": 200, "tp": 0.05, "b1": 1.0},
        # a sample with a spread of its field: 16 isochromats, five pools, whole final states
        {"name": "spread", "kind": "spread", "offsets": 101, "pools": 5, "mt": True, "nodes": 16, "sigma": 12.77,
         "pulses": 20, "samples": 100, "tp": 0.05, "b1": 1.0},
        # a fingerprint dictionary: 30 saturation rows per entry, recovery and CW block each
        {"name": "dictionary", "kind": "dictionary", "entries": 32768, "rows": 30},
        # the quick-start fit over an image: (k, f) of one pool from a ladder of four B1 levels
        {"name": "fit_ladder", "kind": "fit", "voxels": 2048, "offsets": 61, "rungs": 4, "pools": 1, "mt": False,
         "free": 2, "iters": 30, "sigma": 0.002},
        # the five-pool model: six values per voxel
        {"name": "fit_six", "kind": "fit", "voxels": 383, "offsets": 61, "rungs": 4, "pools": 4, "mt": True,
         "free": 6, "iters": 10, "sigma": 0.002},
        # a phantom fit: few samples, shaped pulse trains, three values
        {"name": "fit_train", "kind": "fit_train", "voxels": 7, "offsets": 51, "rungs": 2, "pulses": 10,
         "samples": 100, "tp": 0.05, "iters": 6, "sigma": 0.002},
        # a joint fit over voxels of their own pool counts, offsets and trains, one value shared
        {"name": "fit_joint", "kind": "joint", "voxels": 192, "iters": 12, "sigma": 0.005, "most_pulses": 40},
        # the warm-start network: one training step, and inference over an image
        {"name": "mlp_train", "kind": "mlp_train", "batch": 4096, "n_in": 244, "n_out": 6},
        {"name": "mlp_predict", "kind": "mlp_predict", "rows": 65536, "n_in": 244, "n_out": 6},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cw", "train", "train", "train", "spread", "dictionary", "fit", "fit", "fit_train", "joint",
                       "mlp_train", "mlp_predict"])
    if kind == "cw":
        pools = rng.randint(1, 5)
        return {"kind": kind, "voxels": _log(rng, 1, 1024), "offsets": rng.randint(11, 121), "pools": pools,
                "mt": pools >= 2, "tsat": round(rng.uniform(0.4, 5.0), 2), "b1": round(rng.uniform(0.3, 4.0), 2)}
    if kind == "train":
        pools = rng.randint(1, 5)
        style = rng.choice(["regular", "scanner"])
        return {"kind": kind, "style": style, "precision": rng.choice(["f64", "f64", "mixed", "f32"]),
                "device": rng.random() < 0.3, "voxels": _log(rng, 1, 512), "offsets": rng.randint(21, 121), "pools": pools, "mt": rng.random() < 0.5,
                "pulses": rng.randint(2, 36), "samples": rng.randint(16, 200),
                "tp": round(rng.uniform(0.02, 0.1), 3), "b1": round(rng.uniform(0.15, 4.0), 2)}
    if kind == "spread":
        return {"kind": kind, "offsets": rng.randint(21, 121), "pools": rng.randint(1, 5), "mt": rng.random() < 0.5,
                "nodes": rng.randint(2, 16), "sigma": round(rng.uniform(2.0, 15.0), 2), "pulses": rng.randint(2, 20),
                "samples": rng.randint(16, 200), "tp": round(rng.uniform(0.02, 0.1), 3),
                "b1": round(rng.uniform(0.3, 4.0), 2)}
    if kind == "dictionary":
        return {"kind": kind, "entries": _log(rng, 500, 32768), "rows": rng.randint(8, 40)}
    if kind == "fit":
        six = rng.random() < 0.5
        pools = rng.randint(2, 5) if six else 1
        return {"kind": kind, "voxels": _log(rng, 3, 384 if six else 2048), "offsets": rng.randint(21, 81),
                "rungs": rng.randint(2, 4), "pools": pools, "mt": pools >= 3, "free": 6 if six else 2,
                "iters": rng.randint(8, 10 if six else 30), "sigma": 0.002}
    if kind == "fit_train":
        return {"kind": kind, "voxels": _log(rng, 1, 14), "offsets": rng.randint(31, 61), "rungs": rng.randint(1, 2),
                "pulses": rng.randint(4, 20), "samples": rng.randint(20, 200), "tp": round(rng.uniform(0.02, 0.1), 3),
                "iters": rng.randint(3, 6), "sigma": 0.002}
    if kind == "joint":
        return {"kind": kind, "voxels": _log(rng, 10, 192), "iters": rng.randint(4, 12), "sigma": 0.005,
                "most_pulses": rng.randint(5, 40)}
    if kind == "mlp_train":
        return {"kind": kind, "batch": 128 * _log(rng, 1, 64), "n_in": rng.randint(40, 300), "n_out": rng.randint(2, 8)}
    return {"kind": kind, "rows": _log(rng, 100, 131072), "n_in": rng.randint(40, 300), "n_out": rng.randint(2, 8)}


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
FIELDS = ("water_r1", "water_r2", "water_f", "cest_k", "cest_f", "cest_dw", "cest_r1", "cest_r2", "mt_k", "mt_f",
          "mt_dw", "mt_r1", "mt_r2", "mt_lineshape", "b0", "gamma", "b0_inhom", "rel_b1")


def _tissue(rng, n, pools, mt):
    """n voxels as a dict of float64 arrays, (n,) or (n, pools): seeded, in the benchmark's ranges."""
    one = lambda v: np.full(n, float(v))
    pool = lambda j: np.tile([q[j] for q in POOLS[:pools]], (n, 1)).reshape(n, pools)
    return {"water_r1": 1.0 / rng.uniform(0.8, 2.5, n), "water_r2": 1.0 / rng.uniform(0.03, 0.12, n),
            "water_f": one(1), "cest_k": rng.uniform(10.0, 5000.0, (n, pools)),
            "cest_f": rng.uniform(1e-5, 0.02, (n, pools)), "cest_dw": pool(0), "cest_r1": 1.0 / pool(1),
            "cest_r2": 1.0 / pool(2), "mt_k": one(30 if mt else 0), "mt_f": one(0.05 if mt else 0),
            "mt_dw": one(-2.5 if mt else 0), "mt_r1": one(1 if mt else 0), "mt_r2": one(1e5 if mt else 1),
            "mt_lineshape": one(2 if mt else 0), "b0": one(B0), "gamma": one(GAMMA),
            "b0_inhom": rng.uniform(-0.3, 0.3, n), "rel_b1": rng.uniform(0.9, 1.1, n)}


def _start(p):
    """The start states (n, 3 (1 + pools) + 1)."""
    n, nc = p["cest_k"].shape
    m = np.zeros((n, 3 * nc + 4))
    m[:, 2 * nc + 2] = p["water_f"]
    m[:, 2 * nc + 3:3 * nc + 3] = p["cest_f"]
    m[:, 3 * nc + 3] = p["mt_f"]
    return m


def _table(rows):
    """An event table (type, dt, amp, phase, freq, adc), each (rows, events), from lists of
    (type, dt, amp, phase, freq) per row."""
    a = np.array(rows, np.float64)
    typ = a[:, :, 0].astype(np.int32)
    return (typ,) + tuple(np.ascontiguousarray(a[:, :, j]) for j in range(1, 5)) + (
        np.where(typ == 3, 0, -1).astype(np.int32),)


def _cw(ppm, b1s, tsat):
    amp = lambda b: b * GAMMA / (2 * np.pi)
    return _table([[(1, tsat, amp(b), 0.0, f * HZ_PPM), (3, 0.0, 0.0, 0.0, 0.0)] for b in b1s for f in ppm])


def _shape(n):
    t = (np.arange(n) + 0.5) / n
    s = np.exp(-((t - 0.5) ** 2) / (2 * (1.0 / 6.0) ** 2))
    return s / s.max()


def _train(c, ppm, b1):
    """`regular`: shaped pulses with equal gaps, a spoiler, 3 s recovery, readout (bench.py). `scanner`: a
    recovery first, every pulse with a phase of its own, a spoiler and a delay of its own after it, and a
    slightly skewed shape, as the tables converted from sequence files have them."""
    n, tp = c["samples"], c["tp"]
    amp = b1 * GAMMA / (2 * np.pi) * _shape(n)
    if c.get("style", "regular") == "scanner":
        amp = amp * (1.0 + 0.02 * np.linspace(-1.0, 1.0, n))
    out = []
    for f in np.asarray(ppm) * HZ_PPM:
        row = []
        if c.get("style", "regular") == "scanner":
            row.append((0, 3.0, 0.0, 0.0, 0.0))
            for j in range(c["pulses"]):
                phase = math.fmod(-2 * math.pi * f * tp * j, 2 * math.pi)
                row += [(1, tp / n, a, phase, f) for a in amp]
                spoil = 0.0009 + 0.00005 * j
                row += [(4, spoil, 0.0, 0.0, 0.0), (0, tp - spoil, 0.0, 0.0, 0.0)]
            row[-1] = (4, 0.0065, 0.0, 0.0, 0.0)
        else:
            for j in range(c["pulses"]):
                row += [(1, tp / n, a, 0.0, f) for a in amp] + [(0, 0.1 * tp, 0.0, 0.0, 0.0)]
            row += [(4, 0.0, 0.0, 0.0, 0.0), (0, 3.0, 0.0, 0.0, 0.0)]
        out.append(row + [(3, 0.0, 0.0, 0.0, 0.0)])
    return _table(out)


def _dictionary(c, rng):
    b1 = rng.uniform(0.5, 6.0, c["rows"])
    ev = _table([[(0, 1.0, 0.0, 0.0, 0.0), (1, 1.0, b * GAMMA / (2 * np.pi), 0.0, 3.5 * HZ_PPM), (3, 0.0, 0.0, 0.0, 0.0)]
                 for b in b1])
    e = c["entries"]
    nk = max(2, int(round(e ** 0.4)))
    nf = max(2, int(round(e ** 0.3)))
    nt = max(2, e // (nk * nf))
    jig = lambda: 1.0 + 0.02 * rng.random()
    grid = {"cest_k": np.geomspace(10.0, 5000.0, nk) * jig(), "cest_f": np.geomspace(1e-5, 0.02, nf) * jig(),
            "water_r1": 1.0 / (np.linspace(0.8, 2.5, nt) * jig())}
    base = _tissue(np.random.default_rng(5), 1, 1, True)
    base["water_r2"][:] = 1 / 0.07
    base["b0_inhom"][:] = 0.0
    base["rel_b1"][:] = 1.0
    return base, ev, grid


def _inputs(c, seed):
    """(params, table, m0) of the forward cases."""
    rng = np.random.default_rng([seed, 7])
    if c["kind"] == "cw":
        p = _tissue(rng, c["voxels"], c["pools"], c["mt"])
        return p, _cw(np.linspace(-6, 6, c["offsets"]), [c["b1"]], c["tsat"]), _start(p)
    if c["kind"] == "train":
        p = _tissue(rng, c["voxels"], c["pools"], c["mt"])
        return p, _train(c, np.linspace(-10.0, 10.0, c["offsets"]), c["b1"]), _start(p)
    p = _tissue(rng, 1, c["pools"], c["mt"])
    return p, _train(c, np.linspace(-8.0, 8.0, c["offsets"]), c["b1"]), _start(p)


def _slots(c):
    """(field, index, scale, lo, hi, x0) of a fit's free values."""
    s = [("cest_k", 0, 100.0, 5.0, 6000.0, 300.0), ("cest_f", 0, 1e-3, 1e-6, 0.05, 8e-4)]
    if c["kind"] == "fit_train":
        return s + [("cest_r2", 0, 10.0, 1.0, 200.0, 50.0)]
    if c["kind"] == "joint" or c["free"] == 6:
        s += [("cest_k", 1, 100.0, 5.0, 6000.0, 300.0), ("cest_f", 1, 1e-3, 1e-6, 0.05, 8e-4),
              ("water_r2", None, 10.0, 5.0, 50.0, 1 / 0.07), ("b0_inhom", None, 0.1, -0.5, 0.5, 0.0)]
    if c["kind"] == "joint":
        s += [("water_r1", None, 1.0, 0.2, 2.0, 0.7)]
    return s


def _truth(c, seed):
    """The tissues behind a fit's measurement."""
    rng = np.random.default_rng([seed, 11])
    n = c["voxels"]
    p = _tissue(rng, n, c.get("pools", 1), c.get("mt", False))
    p["water_r1"][:] = 1 / 1.3
    p["rel_b1"][:] = 1.0
    p["cest_k"][:, 0], p["cest_f"][:, 0] = rng.uniform(100.0, 800.0, n), rng.uniform(4e-4, 2e-3, n)
    if c.get("free") == 6:
        p["cest_k"][:, 1], p["cest_f"][:, 1] = rng.uniform(100.0, 800.0, n), rng.uniform(4e-4, 2e-3, n)
        p["cest_k"][:, 2:], p["cest_f"][:, 2:] = 1000.0, 2e-3
        p["water_r2"], p["b0_inhom"] = rng.uniform(9.0, 25.0, n), rng.uniform(-0.2, 0.2, n)
    else:
        p["water_r2"][:] = 1 / 0.07
        p["b0_inhom"][:] = 0.0
    return p


def _fit_problem(c, seed):
    """(base params with the fit's start values, table, m0, measured Z)."""
    p = _truth(c, seed)
    ppm = np.linspace(-6, 6, c["offsets"])
    b1s = [0.5, 1.0, 2.0, 4.0][:c["rungs"]]
    if c["kind"] == "fit":
        ev = _cw(ppm, b1s, 2.0)
    else:
        ev = tuple(np.concatenate(x) for x in zip(*[_train(dict(c, style="scanner"), ppm * 0.7, b) for b in b1s]))
    m0 = _start(p)
    z = _spectra(_dev(p), ev, torch.from_numpy(m0).cuda()).cpu().numpy()
    z = z + c["sigma"] * np.random.default_rng([seed, 13]).standard_normal(z.shape)
    base = {k: v.copy() for k, v in p.items()}
    for f, i, _, _, _, x0 in _slots(c):
        (base[f] if i is None else base[f].T[i])[...] = x0
    return base, ev, m0, z


def _joint_problem(c, seed):
    """Voxels of 1..5 pools, 41 or 61 offsets at two levels, 1..most_pulses block pulses each."""
    rng = np.random.default_rng([seed, 17])
    tables, vox = {}, []
    for _ in range(c["voxels"]):
        nc = int(rng.integers(1, 6))
        p = _tissue(rng, 1, nc, False)
        p["water_r1"][:] = 1 / 1.3
        p["rel_b1"][:] = 1.0
        p["cest_k"][:, :2] = rng.uniform(100.0, 1500.0, min(nc, 2))
        p["cest_f"][:, :2] = rng.uniform(4e-4, 4e-3, min(nc, 2))
        key = (int(rng.choice([41, 61])), int(rng.integers(1, c["most_pulses"] + 1)))
        if key not in tables:
            rows = []
            for b in (1.0, 3.0):
                for f in np.linspace(-6.0, 6.0, key[0]) * HZ_PPM:
                    rows.append([(1, 0.05, b * GAMMA / (2 * np.pi), 0.0, f), (0, 0.005, 0.0, 0.0, 0.0)] * key[1]
                                + [(3, 0.0, 0.0, 0.0, 0.0)])
            tables[key] = _table(rows)
        vox.append((p, key))
    noise = [c["sigma"] * rng.standard_normal(2 * k[0]) for _, k in vox]
    return vox, tables, noise


def _joint_true(vox):
    """Noise-free Z of every voxel of a joint fit, in float64 torch."""
    out = [None] * len(vox)
    for idx, p, f, amp, reps in _joint_groups(vox):
        x = _joint_exp(p, f, amp)
        m = torch.from_numpy(np.concatenate([_start(vox[i][0]) for i in idx])).cuda()
        z = _joint_z(x, m[p["row"]], reps)
        for i in idx:
            out[i] = z[p["vox"] == i].cpu().numpy()
    return out


# ------------------------------------------------------------------------------------------------
# the model in plain torch, float64
# ------------------------------------------------------------------------------------------------
def _dev(p):
    return {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in p.items()}


def _super_lorentzian(delta, t2, w0):
    u = torch.linspace(0.0, 1.0, 101, dtype=torch.float64, device=delta.device)
    q = (3 * u * u - 1).abs().clamp_min(1e-6)

    def direct(d):
        s = torch.zeros_like(d)
        for qi in q:
            s = s + torch.exp(-2 * (d * t2 / qi) ** 2) / qi
        return math.sqrt(2 / math.pi) * t2 * s * math.pi * 0.01
    p0, p1, p2, p3 = -w0 - 300, -w0 - 100, w0 + 100, w0 + 300
    y0, y1, y2, y3 = direct(p0), direct(p1), direct(p2), direct(p3)
    c = ((delta - p1 + 1) / (p2 - p1 + 1)).abs()
    bridge = ((2 * c ** 3 - 3 * c ** 2 + 1) * y1 + (3 * c ** 2 - 2 * c ** 3) * y2
              + (c ** 3 - 2 * c ** 2 + c) * 30 * (y1 - y0) + (c ** 3 - c ** 2) * 30 * (y3 - y2))
    return torch.where(delta.abs() >= w0, direct(delta), bridge)


def _generator(p, amp, phase, freq):
    """[A C; 0 0] of one event for a batch of chains: p holds (B,) and (B, pools) values, the event's
    amplitude [Hz], phase [rad] and frequency [Hz] are (B,)."""
    nc = p["cest_k"].shape[-1]
    N, iy, iz = 3 * nc + 4, nc + 1, 2 * nc + 2
    A = torch.zeros(amp.shape[0], N + 1, N + 1, dtype=torch.float64, device=amp.device)
    wf = 2 * math.pi * freq
    w0 = p["gamma"] * p["b0"]
    off = wf - w0 * p["b0_inhom"]
    w1 = 2 * math.pi * amp * p["rel_b1"]
    wx, wy = w1 * torch.cos(phase), w1 * torch.sin(phase)
    k, f = p["cest_k"], p["cest_f"]
    kf = k * f
    kmf = p["mt_k"] * p["mt_f"]
    cells = []

    def put(i, j, v):
        cells.append((i, j, v))
    r2, r1 = p["water_r2"] + kf.sum(-1), p["water_r1"] + kf.sum(-1) + kmf

    def bloch(x, y, z, r2, r1, d):
        put(x, x, -r2), put(y, y, -r2), put(z, z, -r1)
        put(x, y, d), put(y, x, -d)
        put(x, z, -wy), put(z, x, wy)
        put(y, z, wx), put(z, y, -wx)
    bloch(0, iy, iz, r2, r1, off)
    for i in range(nc):
        d = off - p["cest_dw"][:, i] * w0
        bloch(1 + i, iy + 1 + i, iz + 1 + i, p["cest_r2"][:, i] + k[:, i], p["cest_r1"][:, i] + k[:, i], d)
        for b in (0, iy, iz):
            put(b, b + 1 + i, k[:, i]), put(b + 1 + i, b, kf[:, i])
        put(iz + 1 + i, N, p["cest_r1"][:, i] * f[:, i])
    t2 = 1.0 / p["mt_r2"]
    delta = off - p["mt_dw"] * w0
    g = torch.where(p["mt_f"] > 1e-9, _super_lorentzian(delta, t2, w0), torch.zeros_like(t2)) if bool(
        (p["mt_f"] > 1e-9).any()) else torch.zeros_like(t2)
    put(N - 1, N - 1, -(p["mt_r1"] + p["mt_k"] + w1 * w1 * g))
    put(iz, N - 1, p["mt_k"]), put(N - 1, iz, kmf)
    put(iz, N, p["water_r1"]), put(N - 1, N, p["mt_r1"] * p["mt_f"])
    i = torch.tensor([x[0] for x in cells], device=amp.device)
    j = torch.tensor([x[1] for x in cells], device=amp.device)
    v = torch.stack([x[2] for x in cells], -1)
    return A.index_put((torch.arange(A.shape[0], device=amp.device)[:, None], i[None], j[None]), v)


def _expm(X, most=1 << 27):
    """torch.matrix_exp in pieces of bounded size."""
    step = max(1, most // X.shape[-1] ** 2)
    return torch.cat([torch.matrix_exp(X[a:a + step]) for a in range(0, X.shape[0], step)])


def _chains(p, ev, nodes=None):
    """The params of every (voxel, row) chain, voxel-major, and the row of each."""
    n, rows = p["water_r1"].shape[0], ev[1].shape[0]
    q = {k: v.repeat_interleave(rows, 0) for k, v in p.items()}
    return q, np.tile(np.arange(rows), n)


def _propagate(q, row, ev, m, tangent=None):
    """Final states (B, N) of the chains q (rows `row` of the table ev) from the states m. With `tangent`
    = (dq, dm), a direction of the params and of the states, also the states' derivative."""
    typ, dt, amp, phase, freq, _ = ev
    N = m.shape[-1]
    nc = (N - 4) // 3
    B = m.shape[0]
    col = lambda a, e: torch.from_numpy(a[:, e][row]).cuda()
    memo = {}
    one = torch.ones(B, 1, dtype=torch.float64, device=m.device)
    x = torch.cat([m, one], 1)
    dx = None if tangent is None else torch.cat([tangent[1], 0 * one], 1)
    for e in range(dt.shape[1]):
        if float(np.max(dt[:, e])) > 1e-9:
            key = (amp[:, e].tobytes(), freq[:, e].tobytes(), dt[:, e].tobytes())
            ph = col(phase, e)
            # events that differ in phase only: the same exponential in the frame turned by the phase
            if key not in memo:
                if len(memo) > 400:
                    memo.clear()
                a, f, h = col(amp, e), col(freq, e), col(dt, e)[:, None, None]
                zero = torch.zeros_like(ph)
                X = _generator(q, a, zero, f) * h
                if tangent is None:
                    memo[key] = (_expm(X), None)
                else:
                    dX = torch.func.jvp(lambda *v: _generator(dict(zip(FIELDS, v)), a, zero, f),
                                        tuple(q[k] for k in FIELDS), tuple(tangent[0][k] for k in FIELDS))[1] * h
                    big = torch.zeros(B, 2 * N + 2, 2 * N + 2, dtype=torch.float64, device=m.device)
                    big[:, :N + 1, :N + 1] = X
                    big[:, N + 1:, N + 1:] = X
                    big[:, :N + 1, N + 1:] = dX
                    big = _expm(big)
                    memo[key] = (big[:, :N + 1, :N + 1].clone(), big[:, :N + 1, N + 1:].clone())
            E, dE = memo[key]
            x = _turn(x, -ph, nc)
            if dx is not None:
                dx = _turn(dx, -ph, nc)
                dx = _turn((E @ dx[:, :, None] + dE @ x[:, :, None])[:, :, 0], ph, nc)
            x = _turn((E @ x[:, :, None])[:, :, 0], ph, nc)
        spoil = np.isin(typ[:, e], (2, 4))
        if spoil.any():
            s = torch.from_numpy(spoil[row]).cuda()
            for v in (x, dx):
                if v is not None:
                    v[:, :2 * nc + 2] = torch.where(s[:, None], torch.zeros_like(v[:, :2 * nc + 2]), v[:, :2 * nc + 2])
    return (x[:, :N], None if dx is None else dx[:, :N])


def _turn(x, ph, nc):
    if not bool((ph != 0).any()):
        return x.clone()
    c, s = torch.cos(ph)[:, None], torch.sin(ph)[:, None]
    a, b = x[:, :nc + 1], x[:, nc + 1:2 * nc + 2]
    return torch.cat([c * a - s * b, s * a + c * b, x[:, 2 * nc + 2:]], 1)


def _spectra(p, ev, m0):
    """Z (voxels, rows) of device params p and start states m0."""
    q, row = _chains(p, ev)
    nc = p["cest_k"].shape[1]
    x, _ = _propagate(q, row, ev, m0.repeat_interleave(ev[1].shape[0], 0))
    return x[:, 2 * nc + 2].reshape(p["water_r1"].shape[0], -1)


def _with(base, slots, x):
    """base with the scaled values x (n, P) written in."""
    p = {k: v.clone() for k, v in base.items()}
    for j, (f, i, s, *_) in enumerate(slots):
        (p[f] if i is None else p[f].T[i])[...] = x[:, j] * s
    return p


def _lm(base, ev, m0, z, slots, iters):
    """Per-voxel bounded Levenberg-Marquardt: (x physical, Z at x)."""
    n, P, rows = z.shape[0], len(slots), ev[1].shape[0]
    nc = base["cest_k"].shape[1]
    scale = torch.tensor([s[2] for s in slots], dtype=torch.float64, device=z.device)
    lo, hi = (torch.tensor([s[j] for s in slots], dtype=torch.float64, device=z.device) / scale for j in (3, 4))
    x = (torch.tensor([s[5] for s in slots], dtype=torch.float64, device=z.device) / scale).repeat(n, 1)
    lam = torch.full((n,), 1e-2, dtype=torch.float64, device=z.device)
    m = m0.repeat_interleave(rows, 0)
    eye = torch.eye(P, dtype=torch.float64, device=z.device)
    for _ in range(iters):
        q, row = _chains(_with(base, slots, x), ev)
        J = []
        for f, i, s, *_ in slots:
            dq = {k: torch.zeros_like(v) for k, v in q.items()}
            (dq[f] if i is None else dq[f].T[i])[...] = s
            y, dy = _propagate(q, row, ev, m, (dq, torch.zeros_like(m)))
            J.append(dy[:, 2 * nc + 2].reshape(n, rows))
        r = y[:, 2 * nc + 2].reshape(n, rows) - z
        J = torch.stack(J, -1)
        H, g = J.mT @ J, (J.mT @ r[:, :, None])[:, :, 0]
        A = H + lam[:, None, None] * (torch.diag_embed(torch.diagonal(H, dim1=1, dim2=2)) + 1e-9 * eye)
        t = torch.minimum(torch.maximum(x - torch.linalg.solve(A, g), lo), hi)
        rt = _spectra(_with(base, slots, t), ev, m0) - z
        ok = (rt * rt).sum(1) < (r * r).sum(1)
        x = torch.where(ok[:, None], t, x)
        lam = torch.where(ok, lam * 0.5, lam * 3.0)
    return x * scale, _spectra(_with(base, slots, x), ev, m0)


def _joint_groups(vox):
    """Per pool count: (voxels, chain params, offsets [Hz], amplitudes [Hz], repeats), the chains
    voxel-major; the params also hold each chain's voxel ("vox") and its place in the group ("row")."""
    out = []
    for nc in sorted({v[0]["cest_k"].shape[1] for v in vox}):
        idx = [i for i, v in enumerate(vox) if v[0]["cest_k"].shape[1] == nc]
        rows = [2 * vox[i][1][0] for i in idx]
        rep = np.repeat(np.arange(len(idx)), rows)
        p = _dev({k: np.concatenate([vox[i][0][k] for i in idx])[rep] for k in FIELDS})
        p["vox"], p["row"] = np.array(idx)[rep], rep
        ppm = lambda i: np.tile(np.linspace(-6.0, 6.0, vox[i][1][0]) * HZ_PPM, 2)
        b1 = lambda i: np.repeat([1.0, 3.0], vox[i][1][0]) * GAMMA / (2 * np.pi)
        t = lambda f: torch.from_numpy(np.concatenate([f(i) for i in idx])).cuda()
        out.append((idx, p, t(ppm), t(b1), torch.from_numpy(np.array([vox[i][1][1] for i in idx])[rep]).cuda()))
    return out


def _joint_exp(p, f, amp, dp=None):
    """The propagator of pulse and gap, [P dP; 0 P] with a direction of the params."""
    q = {k: p[k] for k in FIELDS}
    zero = torch.zeros_like(f)
    E = None
    for a, w, h in ((amp, f, 0.05), (zero, zero, 0.005)):
        X = _generator(q, a, zero, w) * h
        if dp is not None:
            dX = torch.func.jvp(lambda *v: _generator(dict(zip(FIELDS, v)), a, zero, w),
                                tuple(q[k] for k in FIELDS), tuple(dp[k] for k in FIELDS))[1] * h
            X = torch.cat([torch.cat([X, dX], 2), torch.cat([torch.zeros_like(X), X], 2)], 1)
        X = _expm(X, 1 << 26)
        E = X if E is None else X @ E
    return E


def _joint_z(P, m, reps):
    """Water z (and with [P dP; 0 P] its derivative) after each chain's own repeats."""
    one = torch.ones(m.shape[0], 1, dtype=torch.float64, device=m.device)
    x = torch.cat([m, one], 1)
    iz = 2 * ((m.shape[1] - 4) // 3) + 2
    if P.shape[1] != x.shape[1]:
        x = torch.cat([torch.zeros_like(x), x], 1)
    for j in range(int(reps.max())):
        x = torch.where((j < reps)[:, None], (P @ x[:, :, None])[:, :, 0], x)
    return x[:, iz] if P.shape[1] == m.shape[1] + 1 else (x[:, m.shape[1] + 1 + iz], x[:, iz])


def _joint_lm(c, vox, z):
    """The joint fit: one damping, every voxel's values and the shared one; (x, shared, rms, cost)."""
    slots = _slots(c)
    PL, n = len(slots) - 1, len(vox)
    sc = torch.tensor([s[2] for s in slots], dtype=torch.float64).cuda()
    lo, hi, x0 = (torch.tensor([s[j] for s in slots], dtype=torch.float64).cuda() / sc for j in (3, 4, 5))
    x, xs, lam = x0[:PL].repeat(n, 1), x0[PL:].clone(), 1e-2
    free = torch.ones(n, PL, dtype=torch.float64).cuda()
    for i, (p, _) in enumerate(vox):
        if p["cest_k"].shape[1] < 2:
            free[i, 2:4] = 0.0
    groups = _joint_groups(vox)
    zs = [torch.from_numpy(np.concatenate([z[i] for i in g[0]])).cuda() for g in groups]
    ms = [torch.from_numpy(np.concatenate([_start(vox[i][0]) for i in g[0]])[g[1]["row"]]).cuda() for g in groups]

    def at(g, x, xs):
        p = {k: (v.clone() if k in FIELDS else v) for k, v in g[1].items()}
        v = torch.from_numpy(p["vox"]).cuda()
        for j, (f, i, s, *_) in enumerate(slots):
            if i is not None and i >= p["cest_k"].shape[1]:
                continue
            (p[f] if i is None else p[f].T[i])[...] = (x[v, j] if j < PL else xs) * s
        return p, v

    def cost(x, xs):
        per = torch.zeros(n, dtype=torch.float64).cuda()
        for g, zm, m in zip(groups, zs, ms):
            p, v = at(g, x, xs)
            per.index_add_(0, v, (_joint_z(_joint_exp(p, g[2], g[3]), m, g[4]) - zm) ** 2)
        return per

    def normal(x, xs):
        H, b = torch.zeros(n, PL + 1, PL + 1, dtype=torch.float64).cuda(), torch.zeros(n, PL + 1, dtype=torch.float64).cuda()
        for g, zm, m in zip(groups, zs, ms):
            p, v = at(g, x, xs)
            J = []
            for f, i, s, *_ in slots:
                if i is not None and i >= p["cest_k"].shape[1]:
                    J.append(torch.zeros_like(zm))
                    continue
                dp = {k: torch.zeros_like(p[k]) for k in FIELDS}
                (dp[f] if i is None else dp[f].T[i])[...] = s
                y, d = _joint_z(_joint_exp(p, g[2], g[3], dp), m, g[4])
                J.append(d)
            J = torch.stack(J, 1)
            H.index_add_(0, v, J[:, :, None] * J[:, None, :])
            b.index_add_(0, v, J * (y - zm)[:, None])
        return H, b
    H, b = normal(x, xs)
    per = cost(x, xs)
    costs = []
    for it in range(c["iters"]):
        Hl = H[:, :PL, :PL] * free[:, :, None] * free[:, None, :]
        d = torch.diagonal(Hl, dim1=1, dim2=2)
        A = Hl + torch.diag_embed(free * lam * (d + 1e-9) + (1 - free))
        hps, gl = H[:, :PL, PL] * free, b[:, :PL] * free
        Y, w = torch.linalg.solve(A, hps), torch.linalg.solve(A, gl)
        hss = H[:, PL, PL].sum()
        ds = -(b[:, PL].sum() - (hps * w).sum()) / (hss + lam * (hss + 1e-9) - (hps * Y).sum())
        t = torch.minimum(torch.maximum(x - (w + Y * ds), lo[:PL]), hi[:PL])
        ts = torch.minimum(torch.maximum(xs + ds, lo[PL:]), hi[PL:])
        pt = cost(t, ts)
        if bool(pt.sum() < per.sum()):
            x, xs, per, lam = t, ts, pt, lam * 0.5
            if it + 1 < c["iters"]:
                H, b = normal(x, xs)
        else:
            lam = lam * 3.0
        costs.append(float(per.sum()))
    X = (x * sc[:PL]).cpu().numpy()
    X[free.cpu().numpy() == 0] = np.nan
    npts = np.array([2 * k[0] for _, k in vox])
    return X, float(xs[0] * sc[PL]), np.sqrt(per.cpu().numpy() / npts), np.array(costs)


# ------------------------------------------------------------------------------------------------
# the network's inputs and its float64 restatement
# ------------------------------------------------------------------------------------------------
def _net_inputs(c, seed):
    rng = np.random.default_rng([seed, 19])
    rows = c.get("batch") or c["rows"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 1)
    x = torch.rand(rows, c["n_in"], generator=g, device="cuda") * 0.8 + 0.1
    t = torch.rand(rows, c["n_out"], generator=g, device="cuda")
    return x, t, rng.uniform(0.3, 0.6, c["n_in"]).astype(np.float32), rng.uniform(2.0, 6.0, c["n_in"]).astype(np.float32)


def _net(c, seed):
    from bmc_b200.warmstart import MLP
    net = MLP(c["n_in"], c["n_out"], 256, 3, seed=seed % 1000)
    x, t, shift, scale = _net_inputs(c, seed)
    net.set_input_normalisation(shift, scale)
    return net, x, t


def _net_exact(c, seed, train):
    """The network of the same start values in float64 (a plain affine - GELU - affine chain)."""
    dims = [c["n_in"], 256, 256, 256, c["n_out"]]
    up = lambda v: (v + 63) // 64 * 64
    pad = [up(dims[0]), 256, 256, 256, up(dims[4])]
    rng = np.random.default_rng(seed % 1000)
    params = []
    for i in range(4):
        b = 1.0 / np.sqrt(dims[i])
        W, v = np.zeros((pad[i + 1], pad[i]), np.float32), np.zeros(pad[i + 1], np.float32)
        W[:dims[i + 1], :dims[i]] = rng.uniform(-b, b, (dims[i + 1], dims[i]))
        v[:dims[i + 1]] = rng.uniform(-b, b, dims[i + 1])
        params += [torch.from_numpy(W).double().cuda(), torch.from_numpy(v).double().cuda()]
    x, t, shift, scale = _net_inputs(c, seed)
    h = torch.zeros(x.shape[0], pad[0], dtype=torch.float64, device="cuda")
    h[:, :dims[0]] = (x.double() - torch.from_numpy(shift).cuda()) * torch.from_numpy(scale).cuda()
    for w in params:
        w.requires_grad_(train)
    for i in range(4):
        h = h @ params[2 * i].T + params[2 * i + 1]
        if i < 3:
            h = 0.5 * h * (1 + torch.erf(h / math.sqrt(2.0)))
    y = h[:, :c["n_out"]]
    if not train:
        return {"y": y}
    loss = ((y - t) ** 2).mean()
    grad = torch.cat([g.reshape(-1) for g in torch.autograd.grad(loss, params)])
    flat = torch.cat([w.detach().reshape(-1) for w in params])
    return {"grad": grad, "params": flat - 1e-3 * grad / (grad.abs() + 1e-8), "loss": loss.detach().reshape(1)}


# ------------------------------------------------------------------------------------------------
# prepare and run
# ------------------------------------------------------------------------------------------------
def _sim_params(p, one=False):
    from bmc_b200.simulation import SimParams
    return SimParams(*[(v[0] if one else v) if k != "mt_lineshape" else (v[0] if one else v).astype(np.int64)
                       for k, v in ((k, p[k]) for k in FIELDS)])


def _spec(c):
    from bmc_b200.fitting import FitSpec, FreeParam
    s = _slots(c)
    return FitSpec([FreeParam(f"v{j}", f, i, sc, lo, hi, x0,
                              scope="shared" if c["kind"] == "joint" and j == len(s) - 1 else "sample")
                    for j, (f, i, sc, lo, hi, x0) in enumerate(s)])


def prepare(case, seed):
    from bmc_b200.fitting import Experiment
    from bmc_b200.simulation import SimEvent
    c, kind = case, case["kind"]
    if kind in ("cw", "train"):
        p, ev, m0 = _inputs(c, seed)
        mz = 2 * c["pools"] + 2
        if c.get("device"):
            return _volume(c, p, ev, m0, mz)
        one = c["voxels"] == 1
        return {"c": c, "exp": Experiment(_sim_params(p, one), SimEvent(*ev), m0[0] if one else m0, mz)}
    if kind == "spread":
        from bmc_b200.simulation import B0Spread
        p, ev, m0 = _inputs(c, seed)
        return {"c": c, "p": _sim_params(p, True), "ev": SimEvent(*ev), "m0": m0[0],
                "spread": B0Spread(c["sigma"], "gauss", c["nodes"])}
    if kind == "dictionary":
        base, ev, grid = _dictionary(c, np.random.default_rng([seed, 23]))
        return {"c": c, "p": _sim_params(base, True), "ev": SimEvent(*ev), "m0": _start(base)[0], "grid": grid}
    if kind in ("fit", "fit_train"):
        base, ev, m0, z = _fit_problem(c, seed)
        return {"c": c, "exp": Experiment(_sim_params(base), SimEvent(*ev), m0, 2 * c.get("pools", 1) + 2),
                "z": z, "spec": _spec(c)}
    if kind == "joint":
        from bmc_b200.uneven import UnevenBatch
        vox, tables, noise = _joint_problem(c, seed)
        tab = {k: SimEvent(*t) for k, t in tables.items()}
        batch = UnevenBatch([Experiment(_sim_params(p, True), tab[k], _start(p)[0], 2 * p["cest_k"].shape[1] + 2)
                             for p, k in vox])
        return {"c": c, "batch": batch, "z": [a + b for a, b in zip(_joint_true(vox), noise)], "spec": _spec(c)}
    net, x, t = _net(c, seed)
    return {"c": c, "net": net, "x": x, "t": t, "loss": torch.zeros(1, device="cuda")}


def _volume(c, p, ev, m0, mz):
    """Device arrays, as a caller of the C interface holds them."""
    from bmc_b200.simulation import DeviceEvents, SimEvent, pack_params, problem
    n, rows = c["voxels"], c["offsets"]
    dev = torch.from_numpy(pack_params(_sim_params(p), n)).cuda()
    events = DeviceEvents(SimEvent(*ev))
    return {"c": c, "pr": problem(n, rows, events.n_events, c["pools"], mz, PRECISION[c["precision"]]), "p": dev,
            "ev": events, "m0": torch.from_numpy(m0).cuda(),
            "out": torch.empty(n, rows, dtype=torch.float64, device="cuda")}


def run(state):
    c, kind = state["c"], state["c"]["kind"]
    if kind == "cw":
        return {"z": state["exp"].simulate()}
    if kind == "train":
        if "pr" in state:
            from bmc_b200.simulation import simulate_device
            simulate_device(state["pr"], state["p"], state["ev"], state["m0"], state["out"])
            return {"z": state["out"]}
        from bmc_b200.simulation import simulate_z
        e = state["exp"]
        return {"z": simulate_z(e.params, e.events, e.m0, e.mz_loc, precision=PRECISION[c["precision"]])}
    if kind == "spread":
        from bmc_b200.simulation import simulate_spectrum_spread
        return {"m": simulate_spectrum_spread(state["p"], state["ev"], state["m0"], c["sigma"], state["spread"])}
    if kind == "dictionary":
        from bmc_b200.mrf import generate_dictionary
        return {"fp": generate_dictionary(state["p"], state["ev"], state["m0"], state["grid"], 4)[1]}
    if kind in ("fit", "fit_train"):
        from bmc_b200.fitting import fit
        r = fit(state["exp"], state["spec"], state["z"], n_iter=c["iters"])
        return {"x": r.x / state["spec"].scales, "z": r.z_fit}
    if kind == "joint":
        from bmc_b200.uneven import fit_joint_uneven
        r = fit_joint_uneven(state["batch"], state["spec"], state["z"], n_iter=c["iters"])
        return {"x": r.x / state["spec"].scales[:-1], "shared": float(r.shared), "rms": r.rms, "cost": r.cost}
    net = state["net"]
    if kind == "mlp_predict":
        return {"y": net.predict(state["x"])}
    state["loss"].zero_()
    net.forward(state["x"], keep=True)
    net.backward(state["t"], state["loss"])
    net.adam(lr=1e-3)
    return {"grad": net.grad, "params": net.params, "loss": state["loss"]}


# ------------------------------------------------------------------------------------------------
# work, tolerance, exact
# ------------------------------------------------------------------------------------------------
def work(case):
    """Bytes: the tables, params and start states once, the results once. Flops of the physics: one
    application of the sparse generator per chain and evolving event (the least that any integrator does), for
    a fit once for the residual, once per tangent and once for the trial point of every iteration."""
    c, kind = case, case["kind"]
    if kind.startswith("mlp"):
        rows = c.get("batch") or c["rows"]
        w = c["n_in"] * 256 + 2 * 256 * 256 + 256 * c["n_out"]
        if kind == "mlp_predict":
            return {"bytes": 4.0 * (rows * (c["n_in"] + c["n_out"]) + w), "flops": 2.0 * rows * w}
        return {"bytes": 4.0 * (rows * (c["n_in"] + c["n_out"]) + 7 * w), "flops": 6.0 * rows * w}
    if kind == "joint":
        chains, events, nnz, P = c["voxels"] * 102.0, c["most_pulses"] + 1.0, 57, 7
        return {"bytes": 8.0 * (chains * 2 + c["voxels"] * 40), "flops": 2.0 * nnz * chains * events * c["iters"] * (P + 2)}
    pools = c.get("pools", 1)
    nnz, N = 12 + 15 * pools, 3 * pools + 4
    if kind == "dictionary":
        return {"bytes": 8.0 * c["entries"] * (13 + 5 + 7) + 4.0 * c["entries"] * c["rows"],
                "flops": 2.0 * nnz * c["entries"] * c["rows"] * 2}
    vox = c.get("voxels", 1)
    rows = c["offsets"] * c.get("rungs", 1)
    evolving = 1 if kind in ("cw", "fit") else c["pulses"] * (c["samples"] + 1) + 1
    table = 44.0 * rows * (evolving + 1)
    chains = vox * rows * c.get("nodes", 1)
    passes = 1 if kind in ("cw", "train", "spread") else c["iters"] * (2 + len(_slots(c)))
    out = vox * rows * (N if kind == "spread" else 1)
    return {"bytes": table + 8.0 * (vox * (13 + 5 * pools + N) + out), "flops": 2.0 * nnz * chains * evolving * passes}


def tolerance(case):
    kind = case["kind"]
    if kind == "cw":
        return {"rel": 1e-10, "max": 1e-9}
    if kind == "train":
        return {"f64": {"rel": 1e-10, "max": 1e-9}, "mixed": {"rel": 1e-8, "max": 1e-7},
                "f32": {"rel": 5e-4, "max": 5e-3}}[case["precision"]]
    if kind == "spread":
        return {"rel": 1e-10, "max": 1e-9}
    if kind == "dictionary":
        return {"rel": 2e-7, "max": 2e-6}
    if kind in ("fit", "fit_train", "joint"):
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 1.2e-2, "max": 0.5}


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind.startswith("mlp"):
        return _net_exact(c, seed, kind == "mlp_train")
    with torch.no_grad():
        if kind in ("cw", "train"):
            p, ev, m0 = _inputs(c, seed)
            if c["voxels"] * c["offsets"] * (c["pulses"] if kind == "train" else 1) > 60000 * 8 or (
                    kind == "train" and c["voxels"] * c["offsets"] > 25000):
                return None
            z = _spectra(_dev(p), ev, torch.from_numpy(m0).cuda())
            return {"z": z[0] if c["voxels"] == 1 and not c.get("device") else z}
        if kind == "spread":
            p, ev, m0 = _inputs(c, seed)
            u, w = np.polynomial.hermite_e.hermegauss(c["nodes"])
            q = {k: np.repeat(v, c["nodes"], 0) for k, v in p.items()}
            q["b0_inhom"] = q["b0_inhom"] + c["sigma"] * u / (GAMMA * B0 / (2 * np.pi))
            ch, row = _chains(_dev(q), ev)
            m = torch.from_numpy(np.repeat(np.repeat(m0, c["nodes"], 0), c["offsets"], 0)).cuda()
            x, _ = _propagate(ch, row, ev, m)
            x = x.reshape(c["nodes"], c["offsets"], -1)
            return {"m": (torch.from_numpy(w / w.sum()).cuda()[:, None, None] * x).sum(0)}
        if kind == "dictionary":
            base, ev, grid = _dictionary(c, np.random.default_rng([seed, 23]))
            mesh = np.meshgrid(*grid.values(), indexing="ij")
            n = mesh[0].size
            p = {k: np.repeat(v, n, 0) for k, v in base.items()}
            for k, v in zip(grid, mesh):
                p[k] = v.reshape(p[k].shape).copy()
            m0 = np.repeat(_start(base), n, 0)
            out = []
            for a in range(0, n, 8192):
                part = _dev({k: v[a:a + 8192] for k, v in p.items()})
                out.append(_spectra(part, ev, torch.from_numpy(m0[a:a + 8192]).cuda()))
            return {"fp": torch.cat(out)}
        if kind in ("fit", "fit_train"):
            if kind == "fit_train" and c["voxels"] * c["samples"] * c["iters"] > 5000:
                return None
            base, ev, m0, z = _fit_problem(c, seed)
            s = _slots(c)
            x, zf = _lm(_dev(base), ev, torch.from_numpy(m0).cuda(), torch.from_numpy(z).cuda(), s, c["iters"])
            return {"x": x / torch.tensor([v[2] for v in s], dtype=torch.float64).cuda(), "z": zf}
        vox, _, noise = _joint_problem(c, seed)
        X, xs, rms, cost = _joint_lm(c, vox, [a + b for a, b in zip(_joint_true(vox), noise)])
        return {"x": X / np.array([s[2] for s in _slots(c)[:-1]]), "shared": xs, "rms": rms, "cost": cost}
