"""The work that users of this framework have it do, as timed cases.

Simulation cases go through `emt6ro.simulation.Experiment` (the reference's
API), `emt6ro.ga_model.EMT6RoModel` (the GA's fitness model) and
`emt6ro.batch.Batch` (ragged batches, recordings); surrogate cases through
`emt6ro.surrogate.Surrogate` and the C ABI's training step on device buffers.

A simulation pass is what a GA generation does with a handle it keeps: reset
to the initial tumours, upload the protocols' doses, run, read the counts.
Passes cover minutes to an hour of simulated time, at the rates of whole runs
of 5 to 20 days: tumours of every size such runs go through are given as
initial states, and part of them has cells under repair from an earlier dose.
"""
from __future__ import annotations

import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "emt6-ro_gb300"))

from emt6ro import _native as N  # noqa: E402
from emt6ro import workloads as wl  # noqa: E402
from emt6ro.batch import Batch  # noqa: E402
from emt6ro.ga_model.model import EMT6RoModel  # noqa: E402
from emt6ro.simulation import Experiment  # noqa: E402
from emt6ro.surrogate import Surrogate  # noqa: E402

SIDE = 51           # interior sites per side of the default lattice
RESOLUTION = 75     # steps per dose bin of the passes below: doses fall inside them
FLOP_PER_SITE = 33  # 3 fields x 11 operations of one diffused site and substep
SUBSTEPS = 23       # over the free sites, and one more over the region of interest
HIDDEN, INPUTS, PADDED = 512, 100, 128


def listed():
    return [
        # one simulation, its whole state read back: interactive use, pure latency
        {"name": "single", "kind": "experiment", "protocols": 1, "tumors": 1, "runs": 1,
         "r_lo": 10, "r_hi": 10, "steps": 300, "repair": False, "state": True},
        # plain simulation: one tumour and protocol, 100 replicates, an hour
        {"name": "plain_100", "kind": "experiment", "protocols": 1, "tumors": 1, "runs": 100,
         "r_lo": 10, "r_hi": 10, "steps": 600, "repair": False, "state": False},
        # the reference-sized GA generation, scored by the fitness model
        {"name": "fitness_2000", "kind": "fitness", "protocols": 20, "tumors": 10, "runs": 10,
         "r_lo": 6, "r_hi": 14, "steps": 300, "repair": True},
        # the GA-scale uniform batch: 20 tumours x 100 protocols x 20 replicates
        {"name": "ga_40000", "kind": "experiment", "protocols": 100, "tumors": 20, "runs": 20,
         "r_lo": 6, "r_hi": 14, "steps": 300, "repair": True, "state": False},
        # the second half of a 10-day horizon: large, regrown tumours
        {"name": "large_tumours", "kind": "experiment", "protocols": 8, "tumors": 19, "runs": 8,
         "r_lo": 15, "r_hi": 24, "steps": 300, "repair": True, "state": False},
        # mixed tumour sizes and horizons over the device work queue
        {"name": "ragged_6000", "kind": "ragged", "sims": 6000, "height": SIDE, "width": SIDE,
         "r_lo": 2, "r_hi": 20, "steps": 600, "mode": 1, "offset": 0},
        # a lattice that is not square, tumours off its centre and against its edges
        {"name": "odd_lattice", "kind": "ragged", "sims": 777, "height": 40, "width": 47,
         "r_lo": 3, "r_hi": 18, "steps": 250, "mode": 0, "offset": 12},
        # recording every step of a few simulations: short launches, one read-back each
        {"name": "timelapse_64", "kind": "timelapse", "sims": 64, "r_lo": 6, "r_hi": 16,
         "steps": 40, "every": 1},
        # surrogate training at its own batch size, and a small one
        {"name": "train_4096", "kind": "train", "batch": 4096, "steps": 4},
        {"name": "train_640", "kind": "train", "batch": 640, "steps": 4},
        # scoring a GA population of 10,000 protocols over 20 tumours, and a generation's 100
        {"name": "score_200000", "kind": "score", "rows": 200_000},
        {"name": "score_2000", "kind": "score", "rows": 2000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["experiment", "experiment", "fitness", "ragged", "ragged", "timelapse",
                       "train", "score"])
    if kind in ("experiment", "fitness"):
        p, t = rng.randint(1, 40), rng.randint(1, 12)
        runs = max(1, _log_int(rng, 1, 12_000) // (p * t))
        lo = rng.randint(2, 22)
        case = {"kind": kind, "protocols": p, "tumors": t, "runs": runs, "r_lo": lo,
                "r_hi": min(24, lo + rng.randint(0, 8)), "steps": rng.randint(100, 600),
                "repair": rng.random() < 0.5}
        if kind == "experiment":
            case["state"] = p * t * runs <= 4
        return case
    if kind == "ragged":
        h, w = rng.choice([(SIDE, SIDE), (SIDE, SIDE), (40, 47), (54, 60)])
        lo = rng.randint(2, 12)
        return {"kind": kind, "sims": _log_int(rng, 50, 6000), "height": h, "width": w,
                "r_lo": lo, "r_hi": min(min(h, w) // 2 - 1, lo + rng.randint(2, 16)),
                "steps": rng.randint(100, 600), "mode": rng.randint(0, 3),
                "offset": rng.choice([0, 0, 6, 13])}
    if kind == "timelapse":
        every = rng.randint(1, 5)
        return {"kind": kind, "sims": _log_int(rng, 1, 600), "r_lo": rng.randint(2, 10),
                "r_hi": rng.randint(10, 22), "steps": every * rng.randint(8, 24), "every": every}
    if kind == "train":
        return {"kind": kind, "batch": 128 * _log_int(rng, 1, 48), "steps": rng.randint(2, 5)}
    return {"kind": kind, "rows": _log_int(rng, 1, 150_000)}


# ---- inputs ------------------------------------------------------------------------
def _lattice(height, width):
    params = wl.default_parameters()
    params.native.lattice_height, params.native.lattice_width = height, width
    return params


def _under_repair(tumor, rng):
    """A third of the cells received 1-4 Gy up to their repair delay ago."""
    s = tumor.sites
    hit = (s["state"] == 1) & (rng.random(s.shape) < 1 / 3)
    n = int(hit.sum())
    irr = rng.integers(4, 17, n).astype(np.float32) * np.float32(0.25)
    delay = (3.3414 * np.exp(0.1492 * irr)).astype(np.float32)
    s["irradiation"][hit] = irr
    s["repair_delay_time"][hit] = delay
    s["time_in_repair"][hit] = delay * rng.uniform(0.02, 1.0, n).astype(np.float32)
    return tumor


def _tumors(params, n, r_lo, r_hi, rng, repair, offset=0):
    native = params.native
    h, w = native.lattice_height, native.lattice_width
    out = []
    for k in range(n):
        r = r_lo + round(k * (r_hi - r_lo) / max(1, n - 1))
        dr, dc = (int(v) for v in rng.integers(-offset, offset + 1, 2))
        center = ((h + 2) // 2 + dr, (w + 2) // 2 + dc)
        t = wl.disc_tumor(params, r, seed=int(rng.integers(1 << 31)), center=center)
        out.append(_under_repair(t, rng) if repair else t)
    return out


def _protocols(n, steps, rng):
    """10 Gy in 1-8 doses inside the pass."""
    slots = max(1, steps // RESOLUTION)
    return [wl.random_protocol(rng, int(rng.integers(1, min(8, slots) + 1)),
                               window_steps=slots * RESOLUTION, grid=RESOLUTION)
            for _ in range(n)]


def _weights(seed):
    """He-scaled weights of the 100 -> 512 -> 512 -> 512 -> 1 network and small
    biases, in the order of Surrogate.SHAPES (input columns padded to 128)."""
    rng = np.random.default_rng(seed)
    out = []
    for fan_in, rows, cols in ((INPUTS, HIDDEN, PADDED), (HIDDEN, HIDDEN, HIDDEN),
                               (HIDDEN, HIDDEN, HIDDEN)):
        w = rng.standard_normal((rows, cols), np.float32) * np.float32(math.sqrt(2 / fan_in))
        w[:, fan_in:] = 0
        out += [w, 0.1 * rng.standard_normal(rows, np.float32)]
    out.append(rng.standard_normal(HIDDEN, np.float32) * np.float32(math.sqrt(2 / HIDDEN)))
    out.append(0.1 * rng.standard_normal(1, np.float32))
    return out


def _rows(n, seed):
    """Raw feature rows: 1-8 doses of 10 Gy in 96 bins, four tumour features."""
    rng = np.random.default_rng(seed)
    protocols = min(n, max(1, n // 20))
    d = np.zeros((protocols, 96), np.float32)
    k = rng.integers(1, 9, protocols)
    share = rng.random((protocols, 8)).astype(np.float32) * (np.arange(8) < k[:, None])
    share = np.round(share / share.sum(1, keepdims=True) * 40) * np.float32(0.25)
    np.add.at(d, (np.arange(protocols)[:, None], rng.integers(0, 96, (protocols, 8))), share)
    t = np.stack([rng.integers(100, 700, 20), rng.uniform(5.5, 14.5, 20),
                  rng.uniform(0.35, 0.55, 20), rng.uniform(8, 14, 20)], 1).astype(np.float32)
    i = np.arange(n)
    return np.concatenate([d[(i // 20) % protocols], t[i % 20]], 1)


_X_MEAN = np.concatenate([np.zeros(96), [330, 10, 0.45, 11]]).astype(np.float32)
_X_STD = np.concatenate([np.full(96, 0.55), [190, 2.6, 0.05, 1.7]]).astype(np.float32)
_Y_MEAN, _Y_STD = 390.0, 115.0


def _batches(case, seed):
    """Standardised training batches and targets, steps x batch rows."""
    rows, batch = case["steps"] * case["batch"], case["batch"]
    x = (_rows(rows, seed + 1) - _X_MEAN) / _X_STD
    rng = np.random.default_rng(seed + 2)
    x = x[rng.permutation(rows)]
    t = 0.4 * np.tanh(x[:, 96] - x[:, :48].sum(1) * 0.3) + 0.5 * rng.standard_normal(rows)
    return (x.reshape(-1, batch, INPUTS).astype(np.float32),
            t.reshape(-1, batch).astype(np.float32))


def _rates(case):
    """Learning rates of the pass: the start of a cosine decay."""
    return [1e-3 * (0.5 + 0.5 * math.cos(math.pi * k / 200)) for k in range(case["steps"])]


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind, s = case["kind"], {"case": case}
    if kind in ("experiment", "fitness"):
        params = _lattice(SIDE, SIDE)
        tumors = _tumors(params, case["tumors"], case["r_lo"], case["r_hi"], rng, case["repair"])
        s["protocols"] = _protocols(case["protocols"], case["steps"], rng)
        if kind == "experiment":
            s["experiment"] = Experiment(params, tumors, case["runs"], case["protocols"],
                                         simulation_steps=case["steps"] + 1,
                                         protocol_resolution=RESOLUTION, seed=seed)
        else:
            s["model"] = EMT6RoModel(params, tumors, case["protocols"], case["runs"],
                                     num_steps=case["steps"], protocol_resolution=RESOLUTION,
                                     seed=seed)
    elif kind in ("ragged", "timelapse"):
        ragged = kind == "ragged"
        params = _lattice(case.get("height", SIDE), case.get("width", SIDE))
        n, kinds = case["sims"], min(case["sims"], 64 if ragged else 8)
        tumors = _tumors(params, kinds, case["r_lo"], case["r_hi"], rng, True,
                         case.get("offset", 0))
        s["protocols"] = _protocols(min(n, 32), case["steps"], rng)
        horizon = None
        if ragged:  # horizons mixed uniformly: a quarter, a half and all of the pass
            horizon = rng.choice([case["steps"] // 4, case["steps"] // 2, case["steps"]], n)
        s["batch"] = Batch(params, tumors, [[] for _ in s["protocols"]], rng.integers(0, kinds, n),
                           rng.integers(0, len(s["protocols"]), n), sim_horizon=horizon,
                           protocol_resolution=RESOLUTION, protocol_length=case["steps"] + 1,
                           seed=seed)
        if ragged:
            s["batch"].set_schedule(case["mode"], 300)
    else:
        rows = case["batch"] if kind == "train" else min(4096, -(-case["rows"] // 128) * 128)
        net = Surrogate(max_batch=rows, seed=seed % 1000)
        net.set_params(_weights(seed))
        net.x_mean, net.x_std, net.y_mean, net.y_std = _X_MEAN, _X_STD, _Y_MEAN, _Y_STD
        s["net"] = net
        if kind == "train":
            x, t = _batches(case, seed)
            s["x"], s["t"] = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
        else:
            s["x"] = _rows(case["rows"], seed + 1)
    return s


# ---- one pass ----------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "experiment":
        e = state["experiment"]
        e.reset()
        e.add_irradiations(state["protocols"])
        e.run(case["steps"])
        out = {"counts": e.get_results()}
        if case["state"]:
            for k, t in enumerate(e.state()):
                out.update({"%d %s" % (k, f): t.sites[f] for f in N.SITE_DTYPE.names})
        return out
    if kind == "fitness":
        return np.asarray(state["model"].predict(state["protocols"]))
    if kind == "ragged":
        b = state["batch"]
        b.reset()
        b.add_irradiations(state["protocols"])
        b.run(case["steps"])
        return {"counts": b.counts(), "summary": b.summary()}
    if kind == "timelapse":
        b = state["batch"]
        b.reset()
        b.add_irradiations(state["protocols"])
        return b.timelapse(case["steps"], case["every"])
    net = state["net"]
    if kind == "score":
        return net.predict(state["x"])
    loss = ctypes.c_float()
    rates = _rates(case)
    for k, lr in enumerate(rates):
        last = ctypes.byref(loss) if k == len(rates) - 1 else None
        N.check(N.lib().emt6_mlp_train_step(net._h, state["x"][k].data_ptr(),
                                            state["t"][k].data_ptr(), case["batch"], lr, last))
    return {"loss": float(loss.value), "params": net.get_params()}


# ---- what a pass cannot do without ---------------------------------------------------
def _site_steps(r, height=SIDE, width=SIDE):
    """Diffused sites of one field and step around a centred disc of radius r:
    the sites closer than r to its centre in every free substep, and the
    region of interest around it in the last one."""
    free = sum(1 for i in range(-r, r + 1) for j in range(-r, r + 1) if i * i + j * j < r * r)
    rows, cols = min(2 * r + 1, height), min(2 * r + 1, width)
    return SUBSTEPS * min(free, rows * cols) + rows * cols


def _sim_work(radii, sims, steps, height=SIDE, width=SIDE):
    """Mean over the radii: state read once and written once (three fields, the
    state byte, 48-byte records of the disc's cells), the stencil's operations."""
    sites = (height + 2) * (width + 2)
    nbytes = sum(2 * (13 * sites + 48 * math.pi * r * r) for r in radii) / len(radii)
    flops = sum(_site_steps(r, height, width) for r in radii) / len(radii) * FLOP_PER_SITE
    return {"bytes": sims * nbytes, "flops": sims * steps * flops}


def work(case):
    kind = case["kind"]
    if kind in ("train", "score"):
        per_row = 2 * (INPUTS * HIDDEN + 2 * HIDDEN * HIDDEN + HIDDEN)
        weights = INPUTS * HIDDEN + 2 * HIDDEN * HIDDEN + 4 * HIDDEN + 1
        if kind == "score":
            return {"bytes": 4 * (case["rows"] * (INPUTS + 1) + weights),
                    "flops": case["rows"] * per_row}
        rows = case["batch"] * case["steps"]
        # forward, weight gradients, and input gradients of all layers but the first;
        # weights and both Adam moments read and written by every step
        return {"bytes": 4 * (rows * (INPUTS + 1) + 6 * weights * case["steps"]),
                "flops": rows * (3 * per_row - 2 * INPUTS * HIDDEN)}
    radii = range(case["r_lo"], max(case["r_lo"], case["r_hi"]) + 1)
    if kind == "ragged":  # horizons of a quarter, a half and all of the steps
        return _sim_work(radii, case["sims"], case["steps"] * 1.75 / 3, case["height"],
                         case["width"])
    if kind == "timelapse":
        return _sim_work(radii, case["sims"], case["steps"])
    return _sim_work(radii, case["protocols"] * case["tumors"] * case["runs"], case["steps"])


# ---- 64-bit values -------------------------------------------------------------------
def _gelu(z):
    return 0.5 * z * (1.0 + torch.erf(z * math.sqrt(0.5)))


def _forward(x, p):
    for k in range(3):
        x = _gelu(x @ p[2 * k].T + p[2 * k + 1])
    return x @ p[6] + p[7]


def exact(case, seed):
    """The surrogate's outputs in 64 bits.  A simulation has none: its counts are
    whole numbers, and its levels follow a path of random decisions."""
    if case["kind"] not in ("train", "score"):
        return None
    p = [torch.from_numpy(a).cuda().double() for a in _weights(seed)]
    p[0] = p[0][:, :INPUTS].contiguous()
    if case["kind"] == "score":
        x = (torch.from_numpy(_rows(case["rows"], seed + 1)).cuda().double()
             - torch.from_numpy(_X_MEAN).cuda().double()) / torch.from_numpy(_X_STD).cuda().double()
        y = torch.cat([_forward(c, p) for c in x.split(8192)])
        return (y * _Y_STD + _Y_MEAN).cpu().numpy()
    xs, ts = (torch.from_numpy(a).cuda().double() for a in _batches(case, seed))
    m, v = [torch.zeros_like(a) for a in p], [torch.zeros_like(a) for a in p]
    for k, lr in enumerate(_rates(case)):
        p = [a.detach().requires_grad_() for a in p]
        loss = ((_forward(xs[k], p) - ts[k]) ** 2).mean()
        grads = torch.autograd.grad(loss, p)
        b1, b2 = 0.9, 0.999
        for i, g in enumerate(grads):
            m[i] = b1 * m[i] + (1 - b1) * g
            v[i] = b2 * v[i] + (1 - b2) * g * g
            step = (m[i] / (1 - b1 ** (k + 1))) / ((v[i] / (1 - b2 ** (k + 1))).sqrt() + 1e-8)
            p[i] = p[i].detach() - lr * step
    w0 = torch.zeros((HIDDEN, PADDED), dtype=torch.float64, device=p[0].device)
    w0[:, :INPUTS] = p[0]
    return {"loss": float(loss), "params": [a.cpu().numpy() for a in [w0, *p[1:]]]}
