"""Performance cases: what users of this framework have it do, through its
public entry points.

One family per hot path, each with the sizes, types and options that path is
used with:

    selfgrav   NBodySelfGrav.step_batch (all-pairs gravity, KDK / Yoshida, f64 / mixed, 2-D / 3-D, tracers)
    frame      NBodyCuda.step_batch (few massive bodies + asteroids, with and without mass)
    ensemble   BatchedSystems.run (thousands of small systems)
    search     broadphase.bounce_suche (asteroid x asteroid candidates of one sample)
    stream     StreamFrames.sample_batch (culling, level of detail, quantisation of a frame)
    mesh2d     NBodyPM.step_batch (isolated 2-D particle mesh)
    mesh3d     PMPeriodic3D.step_batch (periodic 3-D particle mesh, with and without the P3M pair term)

Every scene is drawn from the seed; nothing is read from files.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from solarsystemsimulator_b200 import workloads
from solarsystemsimulator_b200.batched import BatchedSystems
from solarsystemsimulator_b200.broadphase import Erkennungskarte, bounce_suche
from solarsystemsimulator_b200.nbody_kernel import M_MAX, NBodyCuda
from solarsystemsimulator_b200.pm3d import PMPeriodic3D
from solarsystemsimulator_b200.pm_kernel import NBodyPM
from solarsystemsimulator_b200.selfgrav_kernel import NBodySelfGrav
from solarsystemsimulator_b200.stream import LOD_MAX, StreamFrames

DEV = "cuda:0"
G_AU = 4 * math.pi * math.pi
W1 = 1.0 / (2.0 - 2.0 ** (1.0 / 3.0))
W0 = -(2.0 ** (1.0 / 3.0)) / (2.0 - 2.0 ** (1.0 / 3.0))


def listed():
    return [
        # an interactive self-gravitating cloud: a few hundred bodies, 2-D, one film batch of 8 samples;
        # every call is launches and latency
        {"name": "selfgrav cloud 300", "path": "selfgrav", "n": 300, "tracers": 0, "dim": 2, "precision": "mixed",
         "integrator": "kdk", "steps": 8},
        # the film server's self-gravity scene: a few thousand massive bodies carrying test particles
        {"name": "selfgrav 3000 + 20k tracers", "path": "selfgrav", "n": 3000, "tracers": 20000, "dim": 2,
         "precision": "mixed", "integrator": "kdk", "steps": 8},
        # a star cluster in the reference's own precision (f64), 3-D, fourth order; a size that fills no tile
        {"name": "selfgrav f64 cluster 10007", "path": "selfgrav", "n": 10007, "tracers": 0, "dim": 3,
         "precision": "f64", "integrator": "yoshida4", "steps": 1},
        # the benchmark configuration: structure formation, 64^3 sources and 2 x 64^3 tracers
        {"name": "selfgrav structure 262k", "path": "selfgrav", "n": 262144, "tracers": 524288, "dim": 3,
         "precision": "mixed", "integrator": "yoshida4", "steps": 1},
        # the solar system with a main belt of test bodies, one batch of 16 daily samples
        {"name": "frame belt 2000", "path": "frame", "scene": "belt", "asteroids": 2000, "massive": 9, "dim": 3,
         "pair_f32": False, "samples": 16},
        # the asteroid film some hundred samples in, the clouds dispersed over the inner system so that some bodies
        # pass the planets closely: 200,000 asteroids with mass, f32 pair forces, 8 samples, rows on the device
        {"name": "frame film 200k", "path": "frame", "scene": "disc", "asteroids": 200000, "massive": 8, "dim": 2,
         "pair_f32": True, "samples": 8},
        # a parameter study: 4,096 independent systems of 3-64 bodies, 200 steps
        {"name": "ensemble 4096", "path": "ensemble", "systems": 4096, "max_bodies": 64, "steps": 200},
        # collision detection of one film sample of the same clouds
        {"name": "search clouds 200k", "path": "search", "asteroids": 200000, "clouds": 5},
        # the stream server's frame: 8 samples of a million bodies thinned to the client's limit
        {"name": "stream 1M x 8", "path": "stream", "bodies": 1000020, "samples": 8, "log_zoom": False},
        # the reference's particle-mesh dynamics case: 10,000 bodies on a 2048 grid, 4 steps
        {"name": "mesh2d 2048", "path": "mesh2d", "n": 10000, "tracers": 0, "grid": 2048, "steps": 4},
        # the periodic mesh alone: a million particles on 256^3
        {"name": "mesh3d 1M", "path": "mesh3d", "n_side": 128, "mesh": 256, "halos": 0, "short_range": False, "steps": 2},
        # the same particles collapsed into halos, with the P3M pair term (the learned row's mesh method)
        {"name": "mesh3d 1M halos P3M", "path": "mesh3d", "n_side": 128, "mesh": 256, "halos": 400, "short_range": True,
         "steps": 1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["selfgrav", "selfgrav", "frame", "frame", "ensemble", "search", "stream", "mesh2d", "mesh3d",
                       "mesh3d"])
    if path == "selfgrav":
        n = _log_int(rng, 100, 150000)
        tracers = rng.choice([0, _log_int(rng, 10, 2 * n)])
        precision = rng.choice(["mixed", "f64"])
        if precision == "f64":
            n, tracers = min(n, 60000), min(tracers, 60000)
        return {"path": path, "n": n, "tracers": tracers, "dim": rng.choice([2, 3]), "precision": precision,
                "integrator": rng.choice(["kdk", "yoshida4"]), "steps": rng.choice([1, 2, 8]) if n < 20000 else 1}
    if path == "frame":
        scene = rng.choice(["belt", "clouds", "disc"])
        if scene == "belt":
            return {"path": path, "scene": scene, "asteroids": _log_int(rng, 50, 200000), "massive": 9, "dim": 3,
                    "pair_f32": False, "samples": rng.randint(1, 16)}
        return {"path": path, "scene": scene, "asteroids": _log_int(rng, 100, 200000), "massive": rng.randint(2, 12),
                "dim": 2, "pair_f32": rng.choice([True, False]), "samples": rng.randint(1, 8)}
    if path == "ensemble":
        return {"path": path, "systems": _log_int(rng, 32, 4096), "max_bodies": rng.choice([8, 24, 64]),
                "steps": _log_int(rng, 20, 200)}
    if path == "search":
        return {"path": path, "asteroids": _log_int(rng, 500, 200000), "clouds": rng.randint(1, 8)}
    if path == "stream":
        return {"path": path, "bodies": _log_int(rng, 5000, 1000000), "samples": rng.randint(1, 8),
                "log_zoom": rng.choice([True, False])}
    if path == "mesh2d":
        return {"path": path, "n": _log_int(rng, 300, 300000), "tracers": rng.choice([0, _log_int(rng, 100, 20000)]),
                "grid": rng.choice([256, 500, 512, 1000, 1024, 2048, 4096]), "steps": rng.randint(1, 4)}
    side = rng.choice([32, 48, 64, 96, 128])
    return {"path": path, "n_side": side, "mesh": 2 * side, "halos": rng.choice([0, side * 3]),
            "short_range": rng.choice([True, False]), "steps": rng.randint(1, 3)}


# ------------------------------------------------------------------ scenes


def _seed(case, seed):
    """One stream per case and seed, the same in every process."""
    text = "|".join(f"{k}={case[k]}" for k in sorted(case) if k != "name")
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, *text.encode()])


def _disc(rng, n, dim):
    """A uniform disc (ball) of radius 1 in slow rotation."""
    p = rng.normal(0, 1, (dim, n))
    p *= rng.uniform(0, 1, n) ** (1.0 / dim) / np.linalg.norm(p, axis=0)
    v = rng.normal(0, 0.1, (dim, n))
    v[0] -= 0.3 * p[1]
    v[1] += 0.3 * p[0]
    return p, v


def _selfgrav_scene(case, seed):
    rng = _seed(case, seed)
    n, t, dim = case["n"], case["tracers"], case["dim"]
    side = round(n ** (1.0 / 3.0))
    if dim == 3 and n >= 200000 and side ** 3 == n:
        w = workloads.structure_formation(side, t, seed=int(rng.integers(1 << 31)))
        return {"p": w["pos"].T, "v": np.zeros((3, n)), "m": w["mass"], "tp": w["tracer_pos"].T,
                "tv": np.zeros((3, t)), "eps": 1e-3, "dt": 1e-3}
    p, v = _disc(rng, n, dim)
    tp, tv = _disc(rng, t, dim)
    m = np.full(n, 1.0 / n) if case["precision"] == "mixed" else rng.uniform(0.5, 1.5, n) / n
    return {"p": p, "v": v, "m": m, "tp": tp, "tv": tv, "eps": 1e-2, "dt": 1e-3}


def _frame_scene(case, seed):
    """x, v (dim, n), mass, radius, is_ast, G, sample spacing, largest substep."""
    rng = _seed(case, seed)
    n_ast, sub = case["asteroids"], int(rng.integers(1 << 31))
    if case["scene"] == "belt":
        w = workloads.solar_system_belt(n_ast, seed=sub)
        n = len(w["mass"])
        return w["pos"], w["vel"], w["mass"], np.zeros(n), w["is_ast"], w["G"], 1.0, 0.5
    clouds = 5 if n_ast >= 1000 else 1
    per = -(-n_ast // clouds)
    w = workloads.asteroid_clouds(per, clouds, seed=sub)
    m = case["massive"]
    # the star and the planets of the case: a ladder of orbits about 0.4 - 30 AU, the clouds between them
    a = 0.4 * (75.0 ** (np.arange(m - 1) / max(m - 2, 1))) if m > 1 else np.zeros(0)
    th = rng.uniform(0, 2 * np.pi, m - 1)
    pm = np.concatenate([[1.0], 10 ** rng.uniform(-6, -3, m - 1)])
    vc = np.sqrt(w["G"] * (1.0 + pm[1:]) / a)
    pos = np.zeros((2, m + n_ast))
    vel = np.zeros((2, m + n_ast))
    pos[:, 1:m] = a * np.cos(th), a * np.sin(th)
    vel[:, 1:m] = -vc * np.sin(th), vc * np.cos(th)
    if case["scene"] == "clouds":
        pos[:, m:] = w["pos"][:2, 8:8 + n_ast]
        vel[:, m:] = w["vel"][:2, 8:8 + n_ast]
    else:
        r, th = np.sqrt(rng.uniform(1.0, 25.0, n_ast)), rng.uniform(0, 2 * np.pi, n_ast)
        pos[:, m:] = r * np.cos(th), r * np.sin(th)
        vel[:, m:] = np.sqrt(w["G"] / r) * np.array([-np.sin(th), np.cos(th)]) + rng.normal(0, 1e-3, (2, n_ast))
    mass = np.concatenate([pm, w["mass"][8:8 + n_ast]])
    rad = np.concatenate([[0.00465], 10 ** rng.uniform(-5, -4.3, m - 1), w["radius"][8:8 + n_ast]])
    is_ast = np.concatenate([np.zeros(m, np.uint8), np.ones(n_ast, np.uint8)])
    return pos, vel * 365.25, mass, rad, is_ast, G_AU, 0.5 / 365.25, 0.5 / 365.25


def _ensemble_scene(case, seed):
    """An eighth of the systems perturbed figure-8 orbits, the rest planetary
    systems of 3 to max_bodies bodies (log-uniform; the sizes are the case's,
    the orbits the seed's)."""
    rng = _seed(case, seed)
    ns = case["systems"]
    f8 = ns // 8
    sizes = np.round(np.exp(_seed(case, 0).uniform(np.log(3), np.log(case["max_bodies"]), ns - f8))).astype(int)
    sizes = np.clip(sizes, 3, case["max_bodies"])
    k = int((sizes - 1).sum())
    first = np.concatenate([[0], np.cumsum(sizes - 1)])
    owner = np.repeat(np.arange(len(sizes)), sizes - 1)
    a = np.exp(rng.uniform(np.log(0.05), np.log(30.0), k))
    a = a[np.lexsort((a, owner))]
    m = np.exp(rng.uniform(np.log(1e-7), np.log(1e-3), k))
    ang = [rng.uniform(0, 2 * np.pi, k) for _ in range(3)]
    p, v = workloads.kepler_to_cartesian(a, rng.uniform(0, 0.1, k), rng.uniform(0, np.deg2rad(5.0), k), *ang,
                                         G_AU * (1.0 + m))
    out = []
    for _ in range(f8):
        pos, vel, mass = workloads.figure8(rng, 1e-3)
        out.append({"pos": pos, "vel": vel, "mass": mass, "G": 1.0, "dt": 1e-3 * workloads.FIGURE8_PERIOD})
    zero = np.zeros((3, 1))
    for s in range(len(sizes)):
        q = slice(first[s], first[s + 1])
        inner = 2 * np.pi * math.sqrt(a[first[s]] ** 3 / G_AU)
        out.append({"pos": np.concatenate([zero, p[:, q]], 1), "vel": np.concatenate([zero, v[:, q]], 1),
                    "mass": np.concatenate([[1.0], m[q]]), "G": G_AU, "dt": 1e-3 * inner})
    return out


def _stream_scene(case, seed):
    rng = _seed(case, seed)
    n = case["bodies"]
    n_mass, n_inj = min(20, n), n // 10
    x, y = np.zeros(n), np.zeros(n)
    x[:n_mass], y[:n_mass] = rng.uniform(-5, 5, (2, n_mass))
    cen = rng.uniform(-3, 3, (8, 2))
    lab = rng.integers(0, 8, n - n_mass)
    sig = 10 ** rng.uniform(-2.5, -0.3, 8)
    x[n_mass:] = cen[lab, 0] + rng.normal(0, 1, n - n_mass) * sig[lab]
    y[n_mass:] = cen[lab, 1] + rng.normal(0, 1, n - n_mass) * sig[lab]
    is_ast = np.arange(n) >= n_mass
    inj = np.arange(n) >= n - n_inj
    dead = rng.choice(n, n // 50, replace=False)
    vx, vy = rng.normal(0, 1e-3, (2, n))
    xs = [(x + s * vx).astype(np.float32) for s in range(case["samples"])]
    ys = [(y + s * vy).astype(np.float32) for s in range(case["samples"])]
    return xs, ys, is_ast, inj, dead, rng.uniform(-1, 1, len(dead))


def _mesh2d_scene(case, seed):
    rng = _seed(case, seed)
    n, t = case["n"], case["tracers"]
    R, total = 30000.0, 5.6e9
    r, th = R * np.sqrt(rng.uniform(0, 1, n + t)), rng.uniform(0, 2 * np.pi, n + t)
    vvir = math.sqrt(G_AU * total / R)
    ang = rng.uniform(0, 2 * np.pi, n + t)
    return (r * np.cos(th), r * np.sin(th), 0.7 * vvir * np.cos(ang), 0.7 * vvir * np.sin(ang),
            np.full(n, total / n), (R / vvir) / 1000.0)


def _mesh3d_scene(case, seed):
    """A Zel'dovich lattice (face-centred, n_side^3 / 2 particles); with halos,
    70 % of the particles sit in Plummer spheres in equilibrium."""
    rng = _seed(case, seed)
    w = workloads.periodic_structure(case["n_side"], case["mesh"], seed=int(rng.integers(1 << 31)))
    p, n = w["pos"], len(w["pos"])
    v = rng.normal(0, 0.05, (n, 3))
    if case["halos"]:
        share = np.minimum(rng.pareto(1.0, case["halos"]) + 1.0, 120.0)
        home = np.flatnonzero(rng.uniform(0, 1, n) < 0.7)
        h = rng.choice(case["halos"], len(home), p=share / share.sum())
        mass = np.bincount(h, minlength=case["halos"]) / n
        size = 0.15 * (mass / (0.5 / case["halos"])) ** (1.0 / 3.0) / case["halos"] ** (1.0 / 3.0) / 4.0
        d = rng.normal(0, 1, (len(home), 3))
        q = rng.uniform(0, 0.97, len(home)) ** (-2.0 / 3.0) - 1.0
        d *= (size[h] / np.sqrt(np.maximum(q, 1e-9)) / np.linalg.norm(d, axis=1))[:, None]
        p = p.copy()
        p[home] = rng.uniform(0, 1, (case["halos"], 3))[h] + d
        p -= np.floor(p)
        disp = np.sqrt(mass / np.maximum(size, 1e-9) / 10.0)
        v[home] = rng.normal(0, 1, (len(home), 3)) * disp[h][:, None]
    return p, v, 1.0 / n


MESH3D_DT = 1e-4
MESH3D_EPS = 1e-3
P3M = {"r_split_cells": 2.25, "x_cut": 3.0}        # the learned-correction configuration's split


# ----------------------------------------------------------------- prepare


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a)).to(DEV)


def prepare(case, seed):
    path = case["path"]
    if path == "selfgrav":
        s = _selfgrav_scene(case, seed)
        sim = NBodySelfGrav(0, softening_au=s["eps"], G=1.0, integrator=case["integrator"], precision=case["precision"])
        kw = {}
        if case["dim"] == 3:
            kw = {"z": s["p"][2], "vz": s["v"][2], "tracer_z": (s["tp"][2], s["tv"][2])}
        st = sim.load_state(s["p"][0], s["p"][1], s["v"][0], s["v"][1], s["m"],
                            tracer=(s["tp"][0], s["tp"][1], s["tv"][0], s["tv"][1]), **kw)
        return {"case": case, "sim": sim, "st": st, "dt": s["dt"]}
    if path == "frame":
        p, v, m, rad, is_ast, G, dt, sub = _frame_scene(case, seed)
        sim = NBodyCuda(0, G=G, max_sub_dt=sub, pair_f32=case["pair_f32"])
        kw = {"z": p[2], "vz": v[2]} if case["dim"] == 3 else {}
        st = sim.load_state(p[0], p[1], v[0], v[1], m, np.ones(len(m), np.uint8), is_ast, rad, **kw)
        return {"case": case, "sim": sim, "st": st, "dt": dt}
    if path == "ensemble":
        return {"case": case, "ens": BatchedSystems(_ensemble_scene(case, seed))}
    if path == "search":
        rng = _seed(case, seed)
        n = case["asteroids"]
        w = workloads.asteroid_clouds(-(-n // case["clouds"]), case["clouds"], seed=int(rng.integers(1 << 31)))
        card = Erkennungskarte(0, np.ones(n, np.uint8), -np.inf, np.inf)
        vis = rng.uniform(0, 1, n) > 0.02
        card.stammdaten(vis, w["radius"][8:8 + n])
        f = [_dev(a[8:8 + n].astype(np.float32)) for a in (w["pos"][0], w["pos"][1], w["vel"][0], w["vel"][1])]
        return {"case": case, "card": card, "row": f, "r_max": float(w["radius"][8:8 + n].max()),
                "pairs": np.zeros((2, 4 * n), np.int64)}
    if path == "stream":
        xs, ys, is_ast, inj, dead, t_dead = _stream_scene(case, seed)
        sf = StreamFrames(is_ast, inj)
        t = np.full(len(is_ast), np.inf)
        t[dead] = t_dead
        sf.kill_t = torch.minimum(sf.kill_t, _dev(t))
        xs, ys = [_dev(a) for a in xs], [_dev(a) for a in ys]
        view = (0.0, 0.0, -1.0, -1.0) if case["log_zoom"] else (0.0, 0.0, 2.5, 2.5)
        box = sf.box(xs[0], ys[0], view, case["log_zoom"])
        # the frame's payload on the host: per sample the count, u32 indices, u16 x and y
        most, k = min(len(is_ast), 2 * LOD_MAX), case["samples"]
        host = [torch.zeros((k, most), dtype=t).pin_memory() for t in (torch.int32, torch.int16, torch.int16)]
        return {"case": case, "sf": sf, "xs": xs, "ys": ys, "box": box, "host": host, "counts": np.zeros(k, np.int64),
                "times": [0.5 * (k + 1) for k in range(case["samples"])]}
    if path == "mesh2d":
        x, y, vx, vy, m, dt = _mesh2d_scene(case, seed)
        n = case["n"]
        sim = NBodyPM(0, grid_n=case["grid"])
        st = sim.load_state(x[:n], y[:n], vx[:n], vy[:n], m, tracer=(x[n:], y[n:], vx[n:], vy[n:]))
        return {"case": case, "sim": sim, "st": st, "dt": dt}
    p, v, m = _mesh3d_scene(case, seed)
    kw = dict(P3M, short_range=True, softening=MESH3D_EPS) if case["short_range"] else {}
    pm = PMPeriodic3D(case["mesh"], **kw)
    return {"case": case, "sim": pm, "st": pm.load_state(p, v, m)}


# --------------------------------------------------------------------- run


def run(state):
    case = state["case"]
    path = case["path"]
    if path == "selfgrav":
        st = state["st"]
        out = {"rows": state["sim"].step_batch(st, state["dt"], case["steps"])}
        if case["precision"] == "f64":
            d = case["dim"]
            out["x"], out["v"] = st["pos"][st["c"].cur][:, :d], st["vel"][:, :d]
        return out
    if path == "frame":
        st = state["st"]
        if case["asteroids"] >= 50000:          # the film keeps its rows on the device
            out = {"rows": state["sim"].step_batch_device(st, state["dt"], case["samples"])}
        else:
            out = {"rows": state["sim"].step_batch(st, state["dt"], case["samples"])}
        if not case["pair_f32"]:
            out.update(ax=st["ax"], av=st["av"], mx=st["mx"], mv=st["mv"])
        return out
    if path == "ensemble":
        ens = state["ens"]
        ens.run(case["steps"])
        return {"x": ens.x, "v": ens.v}
    if path == "search":
        hits, cand, h, _ = bounce_suche([state["card"]], None, [state["row"]], 0.5, state["r_max"])
        pairs = state["pairs"]
        k = 0 if hits is None else len(hits[0])
        if k:
            pairs[0, :k], pairs[1, :k] = hits
        return {"pairs": pairs, "hits": k, "candidates": cand, "cell": h}
    if path == "stream":
        got = state["sf"].sample_batch(state["xs"], state["ys"], state["times"], 0.5, state["box"], case["log_zoom"],
                                       LOD_MAX)
        for k, sample in enumerate(got):
            m = state["counts"][k] = len(sample[0])
            for host, part in zip(state["host"], sample):
                host[k, :m].copy_(part, non_blocking=True)
        return {"counts": state["counts"], "payload": state["host"]}
    if path == "mesh2d":
        st = state["st"]
        rows = state["sim"].step_batch(st, state["dt"], case["steps"])
        return {"rows": rows, "x": st["x"], "y": st["y"], "vx": st["vx"], "vy": st["vy"]}
    state["sim"].step_batch(state["st"], MESH3D_DT, case["steps"])
    return {"state": state["st"]["buf"][0:6]}


# -------------------------------------------------------------------- work


def work(case):
    """Bytes and operations of one pass that no implementation can avoid; a
    pair interaction counts 20 operations (three differences, r^2, r^-3, three
    sums), an FFT 2.5 N log2 N (real)."""
    path = case["path"]
    if path == "selfgrav":
        ns, nt, d, steps = case["n"], case["n"] + case["tracers"], case["dim"], case["steps"]
        evals = steps * (3 if case["integrator"] == "yoshida4" else 1)
        rows = 4.0 * (2 * d * ns + d * case["tracers"]) * steps
        return {"bytes": 2 * 8.0 * 3 * d * nt + 8.0 * ns + rows, "flops": 20.0 * ns * nt * evals}
    if path == "frame":
        d, n, m, k = case["dim"], case["asteroids"], case["massive"], case["samples"]
        sub = k * (2 if case["scene"] == "belt" else 1)
        both = 1 if case["scene"] == "belt" else 2          # asteroids with mass pull back
        return {"bytes": 2 * 8.0 * 3 * d * n + 4.0 * 2 * d * (n + m) * k, "flops": (60.0 * both + 15.0) * n * m * sub}
    if path == "ensemble":
        logs = (math.log(case["max_bodies"]), math.log(3))
        mean = (case["max_bodies"] - 3) / (logs[0] - logs[1])
        sq = (case["max_bodies"] ** 2 - 9) / (2 * (logs[0] - logs[1]))
        ns = case["systems"]
        return {"bytes": 2 * 48.0 * mean * ns, "flops": 60.0 * case["steps"] * ns * (7 / 8 * (sq - mean) + 6 / 8)}
    if path == "search":
        n = case["asteroids"]
        return {"bytes": 22.0 * n, "flops": 50.0 * n}
    if path == "stream":
        kept = min(LOD_MAX, case["bodies"])
        return {"bytes": case["samples"] * (18.0 * case["bodies"] + 8.0 * kept), "flops": 20.0 * case["bodies"]}
    if path == "mesh2d":
        p, n = 4.0 * case["grid"] ** 2, case["n"] + case["tracers"]
        fft = 2.5 * p * math.log2(p)
        return {"bytes": case["steps"] * (56.0 * n + 8.0 * p + 16.0 * n), "flops": case["steps"] * 3 * fft}
    n, c = case["n_side"] ** 3 / 2, float(case["mesh"]) ** 3
    pairs = 0.0
    if case["short_range"]:
        rc = 2 * P3M["x_cut"] * P3M["r_split_cells"] / case["mesh"]
        pairs = 0.5 * n * n * 4.19 * rc ** 3 * (8.0 if case["halos"] else 1.0)
    return {"bytes": case["steps"] * (2 * 72.0 * n + 8.0 * c + 4 * 8.0 * c),
            "flops": case["steps"] * (4 * 2.5 * c * math.log2(c) + 45.0 * pairs)}


# ------------------------------------------------------------------- exact


def exact(case, seed):
    path = case["path"]
    with torch.no_grad():
        if path == "selfgrav":
            return _exact_selfgrav(case, seed)
        if path == "frame":
            return _exact_frame(case, seed)
        if path == "ensemble":
            return _exact_ensemble(case, seed)
        if path == "mesh2d":
            return _exact_mesh2d(case, seed)
        if path == "mesh3d":
            return _exact_mesh3d(case, seed)
    return None                                  # search and stream return whole numbers


def _pair_sum(tgt, src, gm, eps2):
    """sum_j gm_j (s_j - t_i) / (|s_j - t_i|^2 + eps2)^1.5; tgt (d, T), src (d, S)."""
    out = torch.empty_like(tgt)
    step = max(1, (1 << 26) // src.shape[1])
    for a in range(0, tgt.shape[1], step):
        d = src[:, None, :] - tgt[:, a:a + step, None]
        f = gm * ((d * d).sum(0) + eps2) ** -1.5
        out[:, a:a + step] = (f * d).sum(2)
    return out


def _exact_selfgrav(case, seed):
    n, d, steps = case["n"], case["dim"], case["steps"]
    w = (W1, W0, W1) if case["integrator"] == "yoshida4" else (1.0,)
    if n * (n + case["tracers"]) * (1 + steps * len(w)) > 4e10:
        return None
    s = _selfgrav_scene(case, seed)
    x, v = _dev(np.concatenate([s["p"], s["tp"]], 1)), _dev(np.concatenate([s["v"], s["tv"]], 1))
    gm, eps2, dt = _dev(s["m"]), s["eps"] ** 2, s["dt"]
    a = _pair_sum(x, x[:, :n], gm, eps2)
    rows = []
    for _ in range(steps):
        for c in w:
            v = v + a * (0.5 * c * dt)
            x = x + v * (c * dt)
            a = _pair_sum(x, x[:, :n], gm, eps2)
            v = v + a * (0.5 * c * dt)
        rows.append(torch.cat([x[:, :n].reshape(-1), v[:, :n].reshape(-1), x[:, n:].reshape(-1)]))
    out = {"rows": torch.stack(rows)}
    if case["precision"] == "f64":
        out["x"], out["v"] = x.T.contiguous(), v.T.contiguous()
    return out


def _field(p, q, qm, G, soft):
    """Field of the massive bodies q (d, M) at p (d, n)."""
    d = q[:, None, :] - p[:, :, None]
    r2 = (d * d).sum(0) + soft
    return (G * qm / (r2 * torch.sqrt(r2)) * d).sum(2)


def _encounter(p, v, q, u):
    """Smallest distance / speed / 20 of each column of p, v to the columns of q, u."""
    d, w = q[:, None, :] - p[:, :, None], u[:, None, :] - v[:, :, None]
    dist, speed = (d * d).sum(0).sqrt().clamp_min(1e-12), (w * w).sum(0).sqrt()
    return torch.where(speed > 1e-9, dist / speed / 20.0, torch.inf)


def _exact_frame(case, seed):
    """The frame integrator in plain torch: a substep of the smallest massive
    encounter time, calm asteroids and massive bodies by one Yoshida step, hot
    asteroids by their own adaptive steps against interpolated masses."""
    pos, vel, mass, _, is_ast, G, raster, cap = _frame_scene(case, seed)
    soft, m_sub, K = 1e-6, 8, case["samples"]
    A, M = np.flatnonzero(is_ast != 0), np.flatnonzero(is_ast == 0)
    x, v, am = _dev(pos[:, A]), _dev(vel[:, A]), _dev(mass[A])
    q, u, qm = _dev(pos[:, M]), _dev(vel[:, M]), _dev(mass[M])
    far = torch.full((len(M),), torch.inf, device=DEV, dtype=torch.float64).diag()

    def pull(xa):
        d = q[:, None, :] - q[:, :, None]
        r2 = (d * d).sum(0) + soft
        a = (G * qm / (r2 * torch.sqrt(r2)) * d).sum(2)
        if bool((am != 0).any()):
            d = q[:, None, :] - xa[:, :, None]
            r2 = (d * d).sum(0) + soft
            a = a - (G * am[:, None] / (r2 * torch.sqrt(r2)) * d).sum(1)
        return a

    def fine(p, w, q0, q1, span, t0):
        tau = torch.zeros(p.shape[1], device=DEV, dtype=torch.float64)
        sub = raster / m_sub

        def at(t, pp):
            qq = q0[:, None, :] + (q1 - q0)[:, None, :] * (t / span)[None, :, None]
            d = qq - pp[:, :, None]
            r2 = (d * d).sum(0)
            f = G * qm / ((r2 + soft) * torch.sqrt(r2 + soft))
            return (f * d).sum(2), r2.sqrt().clamp_min(1e-12)

        for _ in range(8000):
            live = tau < span - 1e-15
            if not bool(live.any()):
                break
            a, dist = at(tau, p)
            speed = ((u[:, None, :] - w[:, :, None]) ** 2).sum(0).sqrt()
            step = torch.where(speed > 1e-9, dist / speed / 20.0, torch.inf).amin(1).clamp_max(cap)
            step = step.clamp_min(cap / 1000.0)
            step = torch.minimum(step, span - tau)
            j = torch.floor((t0 + tau) / sub + 1e-9) + 1.0
            rest = j * sub - (t0 + tau)
            step = torch.where((j <= m_sub) & (rest > 0) & (step > rest), rest, step)
            step = torch.where(live, step, torch.zeros_like(step))
            t = tau.clone()
            for c in (W1, W0, W1):
                h = c * step
                p = p + w * h + 0.5 * a * h * h
                t = t + h
                b, _ = at(t, p)
                w = w + 0.5 * (a + b) * h
                a = b
            tau = tau + step
        return p, w

    a, b = _field(x, q, qm, G, soft), pull(x)
    rows = []
    for _ in range(K):
        rem = raster
        while rem > 1e-12:
            step = float((_encounter(q, u, q, u) + far.nan_to_num(nan=0.0, posinf=torch.inf)).min()) if len(M) > 1 else cap
            dt = min(max(min(step, cap), cap / 1000.0), rem)
            t0 = raster - rem
            rem -= dt
            hot = _encounter(x, v, q, u).amin(1) < dt
            calm = ~hot
            q0, xh, vh = q.clone(), x[:, hot], v[:, hot]
            for c in (W1, W0, W1):
                h = c * dt
                x = torch.where(calm, x + v * h + 0.5 * a * h * h, x)
                q = q + u * h + 0.5 * b * h * h
                an = _field(x, q, qm, G, soft)
                v = torch.where(calm, v + 0.5 * (a + an) * h, v)
                a = torch.where(calm, an, a)
                bn = pull(x)
                u = u + 0.5 * (b + bn) * h
                b = bn
            if bool(hot.any()):
                xh, vh = fine(xh, vh, q0, q, dt, t0)
                x[:, hot], v[:, hot] = xh, vh
                a[:, hot] = _field(xh, q, qm, G, soft)
        row = torch.empty((2 * case["dim"], len(mass)), device=DEV, dtype=torch.float64)
        iA, iM = torch.as_tensor(A, device=DEV), torch.as_tensor(M, device=DEV)
        row[:, iA] = torch.cat([x, v])
        row[:, iM] = torch.cat([q, u])
        rows.append(row if case["asteroids"] >= 50000 else row.reshape(-1))
    out = {"rows": torch.stack(rows)}
    if not case["pair_f32"]:
        out.update(ax=x, av=v, mx=q, mv=u)
    return out


def _exact_ensemble(case, seed):
    """Every system padded to the largest, all of them advanced together."""
    systems = _ensemble_scene(case, seed)
    big = max(len(s["mass"]) for s in systems)
    if len(systems) * big * big * case["steps"] > 4e9:
        return None
    ns = len(systems)
    x, v, gm = np.zeros((ns, big, 3)), np.zeros((ns, big, 3)), np.zeros((ns, big))
    for i, s in enumerate(systems):
        k = len(s["mass"])
        x[i, :k], v[i, :k], gm[i, :k] = s["pos"].T, s["vel"].T, s["G"] * s["mass"]
        x[i, k:] = 1e6 + np.arange(big - k)[:, None]
    x, v, gm = _dev(x), _dev(v), _dev(gm)
    dt = _dev(np.array([s["dt"] for s in systems]))[:, None, None]
    off = torch.eye(big, device=DEV, dtype=torch.float64)
    live = (gm > 0).double()[:, :, None]

    def acc(p):
        d = p[:, None, :, :] - p[:, :, None, :]
        r2 = (d * d).sum(3) + off
        return ((gm[:, None, :] * r2 ** -1.5)[..., None] * d).sum(2) * live

    a = acc(x)
    for _ in range(case["steps"]):
        for c in (W1, W0, W1):
            v = v + a * (0.5 * c * dt)
            x = x + v * (c * dt)
            a = acc(x)
            v = v + a * (0.5 * c * dt)
    keep = [torch.as_tensor(np.concatenate([i * big + np.arange(len(s["mass"])) for i, s in enumerate(systems)])).to(DEV)]
    return {"x": x.reshape(-1, 3)[keep[0]].T.contiguous(), "v": v.reshape(-1, 3)[keep[0]].T.contiguous()}


def _exact_mesh2d(case, seed):
    x, y, vx, vy, m, dt = _mesh2d_scene(case, seed)
    n, N, margin = case["n"], case["grid"], 4.0
    p, v, m = _dev(np.stack([x, y])), _dev(np.stack([vx, vy])), _dev(m)
    o = torch.arange(2 * N, device=DEV, dtype=torch.float64)
    o = torch.where(o < N, o, o - 2 * N)

    def accel():
        s = p[:, :n]
        lo, hi = s.amin(1), s.amax(1)
        h = float((hi - lo).max()) / (N - 2 * margin)
        f = (p - (lo - margin * h)[:, None]) / h
        i = f.floor().long().clamp(0, N - 2)
        t = f - i
        corner = [(i[0] + a, i[1] + b, (t[0] if a else 1 - t[0]) * (t[1] if b else 1 - t[1])) for a in (0, 1) for b in (0, 1)]
        rho = torch.zeros(2 * N * 2 * N, device=DEV, dtype=torch.float64)
        for a, b, w in corner:
            rho.index_add_(0, a[:n] * 2 * N + b[:n], m * w[:n])
        rk = torch.fft.rfft2(rho.view(2 * N, 2 * N))
        d = (o[:, None] * h, o[None, :] * h)
        inv = (d[0] ** 2 + d[1] ** 2 + (1.5 * h) ** 2) ** -1.5
        out = []
        for c in (0, 1):
            field = torch.fft.irfft2(rk * torch.fft.rfft2(-G_AU * d[c] * inv), s=(2 * N, 2 * N)).reshape(-1)
            out.append(sum(w * field[a * 2 * N + b] for a, b, w in corner))
        return torch.stack(out)

    a = accel()
    rows = []
    for _ in range(case["steps"]):
        v = v + 0.5 * dt * a
        p = p + dt * v
        a = accel()
        v = v + 0.5 * dt * a
        rows.append(torch.cat([p[0, :n], p[1, :n], v[0, :n], v[1, :n], p[0, n:], p[1, n:]]))
    return {"rows": torch.stack(rows), "x": p[0, :n], "y": p[1, :n], "vx": v[0, :n], "vy": v[1, :n]}


def _exact_mesh3d(case, seed):
    p, v, m = _mesh3d_scene(case, seed)
    n, N = len(p), case["mesh"]
    if case["short_range"] and n > 60000:
        return None
    x, v = _dev(p.T), _dev(v.T)
    rs = (P3M["r_split_cells"] if case["short_range"] else 0.6) / N
    f = torch.fft.fftfreq(N, 1.0 / N, device=DEV, dtype=torch.float64)
    f[N // 2] = N / 2
    half = f[: N // 2 + 1].abs()

    def win(k):
        s = torch.sinc(k / N) ** -4
        return s * torch.exp(-(2 * math.pi * k) ** 2 * rs * rs)

    def odd(k):
        return torch.where(k.abs() == N // 2, 0.0, 2 * math.pi * k)

    k2 = (2 * math.pi) ** 2 * (f[:, None, None] ** 2 + f[None, :, None] ** 2 + half[None, None, :] ** 2)
    k2[0, 0, 0] = 1.0
    green = 4 * math.pi * win(f)[:, None, None] * win(f)[None, :, None] * win(half)[None, None, :] / k2
    green[0, 0, 0] = 0.0
    grad = (odd(f)[:, None, None], odd(f)[None, :, None], odd(half)[None, None, :])

    def accel():
        g = x * N
        i = g.floor()
        t = g - i
        i = i.long() % N
        corner = []
        for a in (0, 1):
            for b in (0, 1):
                for c in (0, 1):
                    at = (((i[0] + a) % N) * N + (i[1] + b) % N) * N + (i[2] + c) % N
                    corner.append((at, (t[0] if a else 1 - t[0]) * (t[1] if b else 1 - t[1]) * (t[2] if c else 1 - t[2])))
        rho = torch.zeros(N ** 3, device=DEV, dtype=torch.float64)
        for at, w in corner:
            rho.index_add_(0, at, w * (m * N ** 3))
        rk = torch.fft.rfftn(rho.view(N, N, N)) * green
        out = []
        for d in range(3):
            field = torch.fft.irfftn(1j * grad[d] * rk, s=(N, N, N)).reshape(-1)
            out.append(sum(w * field[at] for at, w in corner))
        a = torch.stack(out)
        return a + _exact_short(x, m, rs) if case["short_range"] else a

    a = accel()
    for _ in range(case["steps"]):
        v = v + 0.5 * MESH3D_DT * a
        x = x + MESH3D_DT * v
        x = x - x.floor()
        a = accel()
        v = v + 0.5 * MESH3D_DT * a
    return {"state": torch.cat([x, v])}


def _exact_short(x, m, rs):
    alpha = 0.5 / rs
    cut = P3M["x_cut"] / alpha
    out = torch.empty_like(x)
    step = max(1, (1 << 25) // x.shape[1])
    for a in range(0, x.shape[1], step):
        d = x[:, None, :] - x[:, a:a + step, None]
        d = d - d.round()
        r2 = (d * d).sum(0)
        r = r2.sqrt()
        z = alpha * r
        g = torch.erfc(z) + 2.0 / math.sqrt(math.pi) * z * torch.exp(-z * z)
        f = (g - 1.0) / (r2 * r) + (r2 + MESH3D_EPS ** 2) ** -1.5
        f = torch.where((r2 > 0) & (r < cut), m * f, 0.0)
        out[:, a:a + step] = (f * d).sum(2)
    return out


assert M_MAX >= 12, "the frame cases hold at most 12 massive bodies"
