"""The work that programs have this framework do, as cases for timing and for
comparing results: isolated Biot-Savart sums from one wing's call to wakes at
a field grid, whole runs from the case files on, steps of a developed wake
(one rotor, many rotors, coupled rotors), and the surrogate's gradient.

A developed wake is made without running the hundreds of steps that lead to
it: the case is started, its checkpoint's wake arrays are replaced by a
contracting, descending helical sheet behind the wing (perturbed from the
seed), and the checkpoint is loaded at a step past the truncation.

The FP32 precisions' results are handed on as float32, which is what they
carry; the FP64 ones stay float64.
"""
import math
import os
import tempfile

import numpy as np
import torch

from volcanor_gb300 import cases as C
from volcanor_gb300 import lib

PRECISION = {"fp64": lib.PREC_FP64, "fp32": lib.PREC_FP32, "near64": lib.PREC_FP32_NEAR64}
RING_FLOPS = 176.0  # one ring at one target: 4 corner terms of 9, 4 edges of 35
FIL_FLOPS = 44.0
LAYERS = (12, 128, 128, 128, 3)


def listed():
    return [
        # a wing's rings at its own collocation points, arrays on the host: the smallest call, all latency
        {"name": "rings_wing_call", "kind": "rings_host", "precision": "fp64", "n": 52, "m": 52},
        # rings on device buffers in the reference's arithmetic: a verification sum
        {"name": "rings_fp64", "kind": "rings", "precision": "fp64", "n": 6001, "m": 30011},
        # the same sum for production, FP32 pairs
        {"name": "rings_fp32", "kind": "rings", "precision": "fp32", "n": 16411, "m": 200003},
        # and with FP64 near pairs
        {"name": "rings_near64", "kind": "rings", "precision": "near64", "n": 50001, "m": 60013},
        # a tip-vortex wake's filaments at a field grid's cell centres (gridgen), arrays on the host
        {"name": "grid_filaments", "kind": "filaments_host", "precision": "fp64", "n": 2592, "m": 59319},
        # the flat wing from its case file through its first two chords' worth of wake
        {"name": "wing_run", "kind": "run_wing", "precision": "fp64", "nc": 4, "ns": 13, "steps": 40},
        # a 4-blade forward-flight rotor from its case file: AIC, factors, the first steps of a growing wake
        {"name": "rotor_run", "kind": "run_rotor", "precision": "near64", "nb": 4, "ns": 75, "steps": 12},
        # the 2-blade hover rotor with its full 6-revolution wake, production arithmetic
        {"name": "hover_steps", "kind": "hover", "precision": "near64", "ns": 24, "rows": 260, "revs": 6, "steps": 8},
        # the same rotor in the reference's arithmetic
        {"name": "hover_steps_fp64", "kind": "hover", "precision": "fp64", "ns": 24, "rows": 260, "revs": 6, "steps": 1},
        # a sweep of uneven rotors advanced together
        {"name": "sweep_steps", "kind": "sweep", "precision": "near64", "cases": 8, "rings": 160, "revs": 3, "steps": 4},
        # two coupled rotors, one above the other
        {"name": "coaxial_steps", "kind": "coaxial", "precision": "near64", "ns": 8, "rows": 24, "trunc": 30, "steps": 4},
        # the surrogate's training gradient over a batch of solver samples
        {"name": "surrogate_gradient", "kind": "gradient", "n": 20000},
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, even over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rings_host", "rings", "rings", "rings", "filaments_host", "run_wing", "run_rotor", "hover",
                       "hover", "sweep", "coaxial", "gradient"])
    if kind == "rings_host":
        return {"kind": kind, "precision": rng.choice(["fp64", "fp32", "near64"]), "n": _spread(rng, 20, 3000),
                "m": _spread(rng, 20, 3000)}
    if kind == "rings":
        precision = rng.choice(["fp64", "fp32", "near64"])
        if precision == "fp64":
            return {"kind": kind, "precision": precision, "n": _spread(rng, 300, 6000), "m": _spread(rng, 300, 30000)}
        return {"kind": kind, "precision": precision, "n": _spread(rng, 1000, 50000), "m": _spread(rng, 1000, 60000)}
    if kind == "filaments_host":
        return {"kind": kind, "precision": rng.choice(["fp64", "near64"]), "n": _spread(rng, 100, 2500),
                "m": _spread(rng, 1000, 59000)}
    if kind == "run_wing":
        return {"kind": kind, "precision": rng.choice(["fp64", "near64"]), "nc": rng.randint(2, 4),
                "ns": rng.randint(7, 13), "steps": rng.randint(10, 40)}
    if kind == "run_rotor":
        return {"kind": kind, "precision": "near64", "nb": rng.randint(2, 4), "ns": rng.randint(12, 75),
                "steps": rng.randint(6, 12)}
    if kind == "hover":
        precision = rng.choice(["near64", "near64", "fp32", "fp64"])
        revs = rng.randint(3, 6)
        return {"kind": kind, "precision": precision, "ns": rng.randint(10, 24),
                "rows": rng.randint(60, min(260, 72 * revs - 30)), "revs": revs,
                "steps": 1 if precision == "fp64" else rng.randint(4, 8)}
    if kind == "sweep":
        return {"kind": kind, "precision": "near64", "cases": rng.randint(4, 8), "rings": rng.randint(60, 160),
                "revs": rng.randint(2, 3), "steps": 4}
    if kind == "coaxial":
        rows = rng.randint(8, 24)
        return {"kind": kind, "precision": rng.choice(["near64", "fp32"]), "ns": rng.randint(5, 8), "rows": rows,
                "trunc": rows + rng.randint(3, 6), "steps": 4}
    return {"kind": kind, "n": _spread(rng, 1000, 20000)}


# ---- inputs ------------------------------------------------------------------

def _unit(rng, n):
    e = rng.normal(size=(n, 3))
    return e / np.linalg.norm(e, axis=1, keepdims=True)


def _rings(n, m, seed):
    """Rings with corners in the unit cube and edges of 0.005 to 0.05, circulations of
    unit spread, cores of 0.002, and targets in the cube."""
    rng = np.random.default_rng(seed)
    a = rng.uniform(size=(n, 3))
    e1 = _unit(rng, n) * rng.uniform(0.005, 0.05, (n, 1))
    e2 = _unit(rng, n) * rng.uniform(0.005, 0.05, (n, 1))
    corners = np.stack([a, a + e1, a + e1 + e2, a + e2], axis=1)
    return corners, np.full((n, 4), 0.002), rng.normal(size=n), rng.uniform(size=(m, 3))


def _filaments(n, m, seed):
    """A helical tip vortex's filaments with growing cores, and the centres of a field grid around it."""
    rng = np.random.default_rng(seed)
    t = np.arange(n + 1) * math.radians(5.0)
    r = 0.78 + 0.22 * np.exp(-0.3 * t)
    node = np.stack([r * np.cos(t), r * np.sin(t), -2.0 * t / max(t[-1], 1.0)], axis=1)
    node += 0.01 * rng.normal(size=node.shape)
    fc = np.stack([node[1:], node[:-1]], axis=1)
    rvc = np.sqrt(0.004 ** 2 + 1e-7 * np.arange(n))
    side = int(math.ceil(m ** (1.0 / 3.0)))
    g = (np.arange(side) + 0.5) / side
    P = np.stack(np.meshgrid(2.4 * g - 1.2, 2.4 * g - 1.2, -2.2 * g, indexing="ij"), axis=-1).reshape(-1, 3)[:m]
    return fc, rvc, 0.1 * (1.0 + 0.1 * rng.normal(size=n)), np.ascontiguousarray(P)


def _samples(n, seed):
    rng = np.random.default_rng(seed)
    p = [rng.uniform(-1, 1, i * o + o) * np.sqrt(6.0 / (i + o)) for i, o in zip(LAYERS[:-1], LAYERS[1:])]
    for q, o in zip(p, LAYERS[1:]):
        q[-o:] *= 0.1
    X = rng.uniform(-1, 1, (n, LAYERS[0]))
    T = np.sin(X[:, :3] * 2.0) + 0.1 * rng.normal(size=(n, 3))
    return np.concatenate(p).astype(np.float32), X.astype(np.float32), T.astype(np.float32)


def _hover_case(ns, rows, revs, theta0, nt):
    cfg = C.config_text(nt=nt, dt=0.0, density=1.2, kinematicVisc=1.5e-5, fdScheme=3, wakeDissipation=1)
    geo = C.geom_text(nb=2, nc=1, ns=ns, nNwake=rows, span=1.0, rootcut=0.2, chord=0.08, Omega=100.0,
                      shaftAxis=(0.0, 0.0, 1.0), theta0=theta0, velBody=(0.0, 0.0, 0.0), spanSpacing=1, chordSpacing=1,
                      spanwiseCore=0.05, streamwiseCoreVec=0.05, apparentViscCoeff=5.0, wakeTruncateNt=72 * revs,
                      symmetricTau=0, pivotLE=0.25)
    return cfg, geo


def _sweep_cases(n, rings, revs, seed, nt):
    rng = np.random.default_rng(seed)
    out = []
    for i in range(n):
        nb = 2 + i % 3  # blades, rings and wake lengths are the case's own; angles and speeds are drawn
        ns = max(8, int(rings * (0.3 + 0.7 * i / max(n - 1, 1)) / nb))
        mu, radius = rng.uniform(0.0, 0.3), rng.uniform(1.0, 2.0)
        cfg = C.config_text(nt=nt, dt=0.0, density=1.2, kinematicVisc=1.5e-5, fdScheme=3, wakeDissipation=1)
        geo = C.geom_text(nb=nb, nc=1, ns=ns, nNwake=72, span=radius, rootcut=0.2, chord=0.08 * radius, Omega=100.0,
                          shaftAxis=(0.0, 0.0, 1.0), theta0=rng.uniform(2.0, 12.0),
                          velBody=(-mu * 100.0 * radius, 0.0, 0.0), spanSpacing=1, chordSpacing=1, spanwiseCore=0.05,
                          streamwiseCoreVec=0.05, apparentViscCoeff=5.0,
                          wakeTruncateNt=72 * (2 + i % max(revs - 1, 1)), symmetricTau=0, pivotLE=0.25)
        out.append((cfg, geo, (-mu * 100.0 * radius, 0.0, 0.0), 0.08 * radius, 5.0 * 1.5e-5))
    return out


# ---- a developed wake through the checkpoint ------------------------------------

# the arrays of a checkpoint file that hold the wake, by their place in it
NEAR_CORNERS, NEAR_PRED, NEAR_GAM, NEAR_CORE, NEAR_AGE = 11, 12, 13, 14, 15
FAR_ENDS, FAR_PRED, FAR_GAM, FAR_CORE, FAR_CORE0, FAR_LEN0, FAR_LEN, FAR_AGE = 16, 17, 18, 19, 20, 21, 22, 23


def _read_checkpoint(path):
    with open(path, "rb") as f:
        data = f.read()
    nh = int.from_bytes(data[:8], "little")
    head = np.frombuffer(data, np.int64, nh, 8).copy()
    arrays, at = [], 8 + 8 * nh
    while at < len(data):
        size = int.from_bytes(data[at:at + 8], "little")
        arrays.append(np.frombuffer(data, np.uint8, size, at + 8).copy())
        at += 8 + size
    return head, arrays


def _write_checkpoint(path, head, arrays):
    with open(path, "wb") as f:
        f.write(len(head).to_bytes(8, "little") + head.tobytes())
        for a in arrays:
            f.write(a.nbytes.to_bytes(8, "little") + a.tobytes())


def _develop(case, step, vel, chord, visc, seed):
    """Gives a started case a wake as of `step`: every blade's near-wake sheet and far-wake tip
    filaments on a helix that contracts and descends with age, swept by the body's velocity
    `vel`, waviness growing with age, cores grown by diffusion from `chord` / 20."""
    rng = np.random.default_rng(seed)
    nb, ns, nw, nf, nc = (case.geti(k) for k in ("nb", "ns", "nNwake", "nFwake", "nc"))
    fd, path = tempfile.mkstemp(suffix=".ckpt")
    os.close(fd)
    try:
        case.checkpoint_save(path)
        head, arrays = _read_checkpoint(path)
        head[1] = step
        _write_checkpoint(path, head, arrays)
        case.checkpoint_load(path)
        dt, omega, hub = case.get("dt")[0], case.get("Omega")[0], case.get("hub")
        te = np.stack([case.get("vr", b + 1).reshape(ns, nc, 4, 3)[:, -1] for b in range(nb)])  # blade, station, corner
        edge = np.concatenate([te[:, :, 1], te[:, -1:, 2]], axis=1) - hub  # blade, node, xyz
        radius = np.linalg.norm(edge[..., :2], axis=-1).max()
        age = np.arange(nw + nf + 1) * dt
        psi = omega * age
        shrink = 0.78 + 0.22 * np.exp(-0.5 * psi)
        cos, sin = np.cos(-psi), np.sin(-psi)
        x = (edge[:, :, None, 0] * cos - edge[:, :, None, 1] * sin) * shrink
        y = (edge[:, :, None, 0] * sin + edge[:, :, None, 1] * cos) * shrink
        r = np.linalg.norm(edge[..., :2], axis=-1)[:, :, None] / radius
        z = edge[:, :, None, 2] - 0.045 * omega * radius * age * (0.6 + 0.6 * r)
        node = np.stack([x, y, z], axis=-1) - np.asarray(vel) * age[:, None]  # the body was there when it shed
        for _ in range(6):
            k, phase = rng.uniform(0.5, 6.0), rng.uniform(0, 2 * math.pi, 3)
            grow = 0.01 * radius * np.minimum(1.0, psi / (2 * math.pi))
            node += grow[:, None] * np.sin(k * psi[:, None] + phase + 2.0 * r[..., None])
        node += hub
        # rings: corner 1 and 2 at the row's own age, 0 and 3 at the row before
        own, before = np.arange(nw), np.maximum(np.arange(nw) - 1, 0)
        ring = np.stack([node[:, :-1, before], node[:, :-1, own], node[:, 1:, own], node[:, 1:, before]], axis=3)
        span = (np.arange(ns) + 0.5) / ns
        gam = 0.05 * omega * radius * chord * np.sqrt(1 - (2 * span - 1) ** 4) * (1 + 0.02 * rng.normal(size=ns))
        sign = np.sign(np.frombuffer(arrays[0].tobytes()).sum()) or 1.0
        near_gam = np.broadcast_to(sign * gam[:, None], (nb, ns, nw)) * (1 + 0.01 * rng.normal(size=(nb, ns, nw)))
        core2 = (0.05 * chord) ** 2 + 4 * 1.2564 * visc * age
        rows = np.sqrt(core2)[own + 1]
        core = np.broadcast_to(np.stack([rows, rows, rows, np.sqrt(core2)[own]], axis=-1), (nb, ns, nw, 4))
        tip = node[:, -1, nw:]
        ends = np.concatenate([tip[:, 1:], tip[:, :-1]], axis=-1)
        length = np.linalg.norm(tip[:, 1:] - tip[:, :-1], axis=-1)
        far_core = np.broadcast_to(np.sqrt(core2)[nw + 1:], (nb, nf))
        new = {NEAR_CORNERS: ring, NEAR_PRED: ring, NEAR_GAM: near_gam, NEAR_CORE: core,
               NEAR_AGE: np.broadcast_to(age[own + 1], (nb, ns, nw)), FAR_ENDS: ends, FAR_PRED: ends,
               FAR_GAM: np.broadcast_to(near_gam[:, -ns // 4:, -1].max(axis=1, keepdims=True) if sign > 0 else
                                        near_gam[:, -ns // 4:, -1].min(axis=1, keepdims=True), (nb, nf)),
               FAR_CORE: far_core, FAR_CORE0: far_core, FAR_LEN0: length, FAR_LEN: length,
               FAR_AGE: np.broadcast_to(age[nw + 1:], (nb, nf))}
        for place, a in new.items():
            a = np.ascontiguousarray(a, np.float64)
            if a.nbytes == arrays[place].nbytes:
                arrays[place] = a
            elif a.size:
                raise ValueError("checkpoint array %d: %d bytes, expected %d" % (place, arrays[place].nbytes, a.nbytes))
        _write_checkpoint(path, head, arrays)
        case.checkpoint_load(path)
    finally:
        os.unlink(path)


# ---- the passes -------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    s = dict(case)
    rng = np.random.default_rng([seed, 7])
    if kind in ("rings_host", "rings"):
        data = _rings(case["n"], case["m"], seed)
        if kind == "rings":
            data = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in data]
            s["V"] = torch.empty_like(data[3])
        s["data"] = data
    elif kind == "filaments_host":
        s["data"] = _filaments(case["n"], case["m"], seed)
    elif kind == "run_wing":
        s["cfg"] = C.config_text(nt=case["steps"], dt=0.025, density=1.0, fdScheme=1, wakeDissipation=0)
        s["geo"] = C.geom_text(nb=1, nc=case["nc"], ns=case["ns"], nNwake=case["steps"], span=4.0, rootcut=0.0,
                               chord=1.0, Omega=0.0, theta0=float(rng.uniform(3, 8)), velBody=(-10.0, 0.0, 0.0),
                               spanSpacing=2, chordSpacing=1, spanwiseCore=0.03, streamwiseCoreVec=0.03,
                               apparentViscCoeff=5.0, symmetricTau=1)
    elif kind == "run_rotor":
        s["cfg"] = C.config_text(nt=72, dt=0.0, density=1.2, kinematicVisc=1.5e-5, fdScheme=3, wakeDissipation=1)
        s["geo"] = C.geom_text(nb=case["nb"], nc=1, ns=case["ns"], nNwake=72, span=2.0, rootcut=0.2, chord=0.12,
                               Omega=100.0, shaftAxis=(0.0, 0.0, 1.0), theta0=float(rng.uniform(6, 11)),
                               velBody=(-20.0, 0.0, 0.0), phiThetaPsi=(0.0, -4.0, 0.0), spanSpacing=1, chordSpacing=1,
                               spanwiseCore=0.05, streamwiseCoreVec=0.05, apparentViscCoeff=5.0, symmetricTau=0,
                               pivotLE=0.25)
    elif kind == "hover":
        at = 72 * case["revs"] + 8
        cfg, geo = _hover_case(case["ns"], case["rows"], case["revs"], float(rng.uniform(7, 9)),
                               at + (500 if case["precision"] == "fp64" else 5000))
        s["case"] = lib.Case(cfg, geo, precision=PRECISION[case["precision"]])
        s["case"].start()
        _develop(s["case"], at, (0.0, 0.0, 0.0), 0.08, 5.0 * 1.5e-5, seed)
    elif kind == "sweep":
        at = 72 * max(case["revs"], 2) + 8
        all_ = _sweep_cases(case["cases"], case["rings"], case["revs"], seed, at + 1600)
        s["case"] = lib.Batch([(cfg, geo, "") for cfg, geo, *_ in all_], precision=PRECISION[case["precision"]])
        s["case"].start()
        for i, (_, _, vel, chord, visc) in enumerate(all_):
            _develop(s["case"].case(i), at, vel, chord, visc, seed + i)
    elif kind == "coaxial":
        sc = C.rotor_pair(nt=case["trunc"] + 6000, ns=case["ns"], n_nwake=case["rows"], truncate_nt=case["trunc"],
                          theta0=float(rng.uniform(7, 9)))
        s["case"] = lib.System(sc.config, sc.geoms, precision=PRECISION[case["precision"]])
        s["case"].start()
        s["case"].step(case["trunc"] + 2)
    elif kind == "gradient":
        p, s["X"], s["T"] = _samples(case["n"], seed)
        s["net"] = lib.Mlp(LAYERS)
        s["net"].set_params(p)
    else:
        raise ValueError(kind)
    return s


def _state(case, blades, precision):
    """What a program that follows a run keeps after some steps: circulations and wakes."""
    out = {"gam": case.get("gamVec")}
    for b in blades:
        for name, a in zip(("rings", "rings_gam", "far", "far_gam"), case.get_wake(b)):
            out["%s%d" % (name, b)] = a
    return _own(out, precision)


def _own(v, precision):
    """FP32 results as float32."""
    if precision == "fp64":
        return v
    return {k: _own(x, precision) for k, x in v.items()} if isinstance(v, dict) else v.astype(np.float32)


def run(s):
    kind, precision = s["kind"], s.get("precision")
    if kind == "rings_host":
        return _own(lib.biot_savart_rings(*s["data"], PRECISION[precision]), precision)
    if kind == "filaments_host":
        return _own(lib.biot_savart_filaments(*s["data"], PRECISION[precision]), precision)
    if kind == "rings":
        corners, rvc, gam, P = s["data"]
        lib.biot_savart_rings_device(corners.data_ptr(), rvc.data_ptr(), gam.data_ptr(), s["n"], P.data_ptr(), s["m"],
                                     s["V"].data_ptr(), PRECISION[precision],
                                     torch.cuda.current_stream().cuda_stream)
        return s["V"] if precision == "fp64" else s["V"].to(torch.float32)
    if kind in ("run_wing", "run_rotor"):
        case = lib.Case(s["cfg"], s["geo"], precision=PRECISION[precision])
        case.start()
        case.step(s["steps"])
        out = {"ct": _own(case.ct_hist(), precision), "state": _state(case, range(1, s.get("nb", 1) + 1), precision)}
        case.close()
        return out
    if kind == "hover":
        rows = s["case"].step(s["steps"])
        return {"ct": _own(rows, precision), "state": _state(s["case"], (1, 2), precision)}
    if kind == "sweep":
        rows = s["case"].step(s["steps"])
        gam = {str(i): s["case"].case(i).get("gamVec") for i in range(s["cases"])}
        last = s["case"].case(s["cases"] - 1)
        return {"ct": _own(rows, precision), "gam": _own(gam, precision),
                "last": _state(last, (1,), precision)}
    if kind == "coaxial":
        rows = s["case"].step(s["steps"])
        return {"ct": _own(rows, precision), "states": {str(i): _state(c, (1, 2), precision)
                                                        for i, c in enumerate(s["case"].rotors)}}
    g, loss = s["net"].gradient(s["X"], s["T"])
    return {"gradient": g, "loss": np.float32(loss)}


# ---- the work a pass cannot do without -----------------------------------------------

def _step_work(nb, ns, rows, far, steps, panels):
    """Pairs of one evaluation per step at every wake node (what a predictor's second one changes
    is small) and at the panels, in flops; the wake read and written once per step, in bytes."""
    nodes = nb * (rows * (ns + 1) + far)
    rings, fils = nb * rows * ns, nb * (far + (ns if far else 0))
    pairs = (rings + panels) * nodes + rings * panels
    return {"flops": steps * (RING_FLOPS * pairs + FIL_FLOPS * fils * (nodes + panels)),
            "bytes": steps * 8.0 * (2 * 18 * rings + 2 * 12 * nb * far + 6 * nodes)}


def work(case):
    kind = case["kind"]
    if kind in ("rings_host", "rings"):
        n, m = case["n"], case["m"]
        return {"flops": RING_FLOPS * n * m, "bytes": 8.0 * (17 * n + 6 * m)}
    if kind == "filaments_host":
        n, m = case["n"], case["m"]
        return {"flops": FIL_FLOPS * n * m, "bytes": 8.0 * (8 * n + 6 * m)}
    if kind == "gradient":
        weights = sum(i * o for i, o in zip(LAYERS[:-1], LAYERS[1:]))
        return {"flops": 6.0 * weights * case["n"], "bytes": 4.0 * (15 * case["n"] + 2 * weights)}
    if kind in ("run_wing", "run_rotor"):
        nb = case.get("nb", 1)
        panels = nb * case["ns"] * case.get("nc", 1)
        each = [_step_work(nb, case["ns"], k, 0, 1, panels) for k in range(1, case["steps"] + 1)]
        return {"flops": sum(w["flops"] for w in each) + 2.0 * panels ** 3 + RING_FLOPS * panels ** 2,
                "bytes": sum(w["bytes"] for w in each) + 16.0 * panels ** 2}
    if kind == "hover":
        return _step_work(2, case["ns"], case["rows"], 72 * case["revs"] - case["rows"], case["steps"], 2 * case["ns"])
    if kind == "coaxial":  # every node against both rotors' wakes
        return _step_work(4, case["ns"], case["rows"], case["trunc"] - case["rows"], case["steps"], 4 * case["ns"])
    total = {"flops": 0.0, "bytes": 0.0}
    for i in range(case["cases"]):
        nb = 2 + i % 3
        ns = max(8, int(case["rings"] * (0.3 + 0.7 * i / max(case["cases"] - 1, 1)) / nb))
        w = _step_work(nb, ns, 72, 72 * (1 + i % max(case["revs"] - 1, 1)), case["steps"], nb * ns)
        total = {k: total[k] + w[k] for k in total}
    return total


# ---- values in 64 bits -------------------------------------------------------------------

def _filament_sum(ends, P):
    """Vatistas (n = 2) velocity of filaments (start, end, core, circulation) at P."""
    a, b, core, gam = ends
    V = torch.zeros_like(P)
    px, py, pz = (P[:, k:k + 1] for k in range(3))
    block = max(1, 4_000_000 // max(1, P.shape[0]))
    for i in range(0, a.shape[0], block):
        A, B, w = a[i:i + block], b[i:i + block], gam[i:i + block] * (0.25 / math.pi)
        x1, y1, z1 = (p - A[:, k] for k, p in enumerate((px, py, pz)))
        x2, y2, z2 = (p - B[:, k] for k, p in enumerate((px, py, pz)))
        e = B - A
        cx, cy, cz = y1 * z2 - z1 * y2, z1 * x2 - x1 * z2, x1 * y2 - y1 * x2
        c2 = cx * cx + cy * cy + cz * cz
        d = (e[:, 0] * x1 + e[:, 1] * y1 + e[:, 2] * z1) / torch.sqrt(x1 * x1 + y1 * y1 + z1 * z1)
        d -= (e[:, 0] * x2 + e[:, 1] * y2 + e[:, 2] * z2) / torch.sqrt(x2 * x2 + y2 * y2 + z2 * z2)
        f = w * d / torch.sqrt((core[i:i + block] ** 2 * (e * e).sum(1)) ** 2 + c2 * c2)
        f = torch.where(c2 > 4.930380657631324e-32, f, torch.zeros_like(f))
        V[:, 0] += (f * cx).sum(1)
        V[:, 1] += (f * cy).sum(1)
        V[:, 2] += (f * cz).sum(1)
    return V


def exact(case, seed):
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev, torch.float64)
    if kind in ("rings_host", "rings"):
        corners, rvc, gam, P = (up(a) for a in _rings(case["n"], case["m"], seed))
        a, b = corners.reshape(-1, 3), corners[:, [1, 2, 3, 0]].reshape(-1, 3)
        return _filament_sum((a, b, rvc.reshape(-1), gam.repeat_interleave(4)), P)
    if kind == "filaments_host":
        fc, rvc, gam, P = (up(a) for a in _filaments(case["n"], case["m"], seed))
        return _filament_sum((fc[:, 0], fc[:, 1], rvc, gam), P)
    if kind == "gradient":
        p, X, T = (up(a) for a in _samples(case["n"], seed))
        p.requires_grad_(True)
        h, at = X, 0
        for l, (i, o) in enumerate(zip(LAYERS[:-1], LAYERS[1:])):
            h = h @ p[at:at + i * o].reshape(o, i).T + p[at + i * o:at + i * o + o]
            at += i * o + o
            if l < len(LAYERS) - 2:
                h = torch.tanh(h)
        loss = ((h - T) ** 2).mean()
        loss.backward()
        return {"gradient": p.grad, "loss": float(loss)}
    return None
