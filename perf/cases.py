"""The workloads that this library's speed is measured on.

Each case is one call (or one short sequence of calls) of the public API as a sampling program
makes it: a Markov-chain walk of one of the five models from an extremal tiling, one exact
sample by coupling from the past, one look-back of device-resident coupled chains, or a batch
of exact samples.  Domains and start states are fixed by the sizes, as they are in use; the
randomness of a pass comes from its seed.  Every output is a whole number.

listed() names the cases, draw(rng) gives others of the same ranges, prepare(case, seed) makes
what a program holds before the call, run(state) is one pass, work(case) the bytes and
operations that the pass cannot do without.
"""
import math
import random
from pathlib import Path

import numpy as np
import torch

import randomtilingspublic_gb300 as rt

TUNE_TABLE = Path(rt.__file__).resolve().parent / "tune" / "gb300.txt"


def listed():
    return [
        # The smallest call: a demonstration-sized diamond, a few hundred half-sweeps.  Set-up
        # and launch latency of one Walk.
        {"name": "walk_aztec16", "kind": "domino_walk", "domain": "aztec", "rows": 16, "cols": 16, "steps": 200,
         "rule": "plain", "rng": "tinymt", "table": False, "a": 0.7, "b": 1.0},
        # The minimal domino example's shape: order 100, 10^4 sweeps in the reference's random
        # streams.
        {"name": "walk_aztec100", "kind": "domino_walk", "domain": "aztec", "rows": 100, "cols": 100, "steps": 20000,
         "rule": "cftp", "rng": "tinymt", "table": False, "a": 0.7, "b": 1.0},
        # A ragged rectangle under the two-periodic rule with the counter-based random mode.
        {"name": "walk_rect301x442", "kind": "domino_walk", "domain": "rectangle", "rows": 301, "cols": 442,
         "steps": 6000, "rule": "twoperiodic", "rng": "fast", "table": False, "a": 0.7, "b": 1.0},
        # The benchmark's step: coupled extremal chains of the order-1024 diamond at a = 1,
        # b = 0.5, one look-back of 2^10 sweeps on the device, then both chains' height
        # functions (a chain's whole state) in device memory.
        {"name": "coupled_aztec1024", "kind": "domino_coupled", "order": 1024, "steps": 2048, "rng": "tinymt", "a": 1.0,
         "b": 0.5},
        # One exact uniform sample of a mid-size diamond, look-back doubling until it coalesces.
        {"name": "cftp_aztec40", "kind": "domino_cftp", "order": 40, "rule": "cftp", "rng": "fast", "first": 256,
         "a": 1.0, "b": 1.0},
        # A lozenge walk on the a = b = c = 512 hexagon in the reference's random streams.
        {"name": "walk_hex512", "kind": "lozenge_walk", "side": 512, "steps": 3000, "rng": "tinymt", "q": 0.0},
        # One exact lozenge sample on a small hexagon.
        {"name": "cftp_hex20", "kind": "lozenge_cftp", "side": 20, "first": 128, "rng": "fast", "q": 0.0},
        # A rectangle-triangle walk (this model has walks only).
        {"name": "walk_recttri100", "kind": "recttri_walk", "side": 100, "steps": 3000, "rng": "tinymt", "weighted": False},
        # Bibone tilings of the 512 x 512 rhombus from the brick start.
        {"name": "walk_bibone512", "kind": "bibone_walk", "domain": "rhombus", "rows": 512, "cols": 512, "steps": 6000,
         "rng": "fast"},
        # Six-vertex model, domain-wall boundary, n = 512, a = b = 1, c = 1.5.
        {"name": "walk_sixvertex512", "kind": "six_walk", "n": 512, "sweeps": 2000, "a": 1.0, "b": 1.0, "c": 1.5},
        # One exact six-vertex sample.
        {"name": "cftp_sixvertex48", "kind": "six_cftp", "n": 48, "first": 64, "a": 1.0, "b": 1.0, "c": 1.5},
        # Many exact samples of mixed models and sizes in one call.
        {"name": "batch512", "kind": "batch", "count": 512, "order_lo": 16, "order_hi": 48, "side_lo": 8, "side_hi": 32,
         "b_lo": 0.9},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["domino_walk", "domino_walk", "domino_coupled", "domino_cftp", "lozenge_walk", "lozenge_cftp",
                       "recttri_walk", "bibone_walk", "six_walk", "six_cftp", "batch"])
    mode = rng.choice(["tinymt", "fast"])
    if kind == "domino_walk":
        rule = rng.choice(["plain", "cftp", "twoperiodic"])
        domain = rng.choice(["aztec", "rectangle"])
        rows = _log(rng, 8, 500)
        cols = rows if domain == "aztec" else _log(rng, 8, 500)
        if domain == "rectangle" and rows * cols % 2:
            cols += 1
        return {"kind": kind, "domain": domain, "rows": rows, "cols": cols, "steps": _log(rng, 200, 12000), "rule": rule,
                "rng": mode, "table": mode == "tinymt" and rng.random() < 0.3, "a": round(rng.uniform(0.5, 1.0), 2),
                "b": 1.0}
    if kind == "domino_coupled":
        return {"kind": kind, "order": _log(rng, 32, 1024), "steps": 2 * _log(rng, 128, 1024), "rng": mode, "a": 1.0,
                "b": round(rng.uniform(0.3, 1.0), 2)}
    if kind == "domino_cftp":
        order = _log(rng, 8, 40)
        weighted = order <= 24 and rng.random() < 0.5
        return {"kind": kind, "order": order, "rule": "cftp_twoperiodic" if weighted else "cftp", "rng": mode,
                "first": 2 * _log(rng, 32, 256), "a": 1.0, "b": round(rng.uniform(0.8, 1.0), 2) if weighted else 1.0}
    if kind == "lozenge_walk":
        return {"kind": kind, "side": _log(rng, 8, 512), "steps": _log(rng, 200, 3000), "rng": mode,
                "q": rng.choice([0.0, 0.0, 0.99])}
    if kind == "lozenge_cftp":
        return {"kind": kind, "side": _log(rng, 4, 20), "first": _log(rng, 32, 256), "rng": mode, "q": 0.0}
    if kind == "recttri_walk":
        return {"kind": kind, "side": _log(rng, 4, 256), "steps": _log(rng, 200, 3000), "rng": mode,
                "weighted": rng.random() < 0.5}
    if kind == "bibone_walk":
        domain = rng.choice(["rhombus", "icecream"])
        rows = _log(rng, 10, 512)
        cols = 2 * _log(rng, 5, 256) if domain == "rhombus" else rng.randint(0, rows // 3)
        return {"kind": kind, "domain": domain, "rows": rows, "cols": cols, "steps": _log(rng, 200, 6000), "rng": mode}
    if kind == "six_walk":
        return {"kind": kind, "n": _log(rng, 16, 1024), "sweeps": _log(rng, 100, 1000), "a": round(rng.uniform(0.7, 1.5), 2),
                "b": round(rng.uniform(0.7, 1.5), 2), "c": round(rng.uniform(0.7, 2.0), 2)}
    if kind == "six_cftp":
        a, b = round(rng.uniform(0.8, 1.0), 2), round(rng.uniform(0.8, 1.0), 2)
        return {"kind": kind, "n": _log(rng, 8, 48), "first": _log(rng, 16, 128), "a": a, "b": b,
                "c": round(rng.uniform(1.0, 1.6), 2)}
    return {"kind": kind, "count": _log(rng, 32, 512), "order_lo": 8, "order_hi": rng.randint(16, 48), "side_lo": 4,
            "side_hi": rng.randint(8, 32), "b_lo": round(rng.uniform(0.9, 1.0), 2)}


def _domino_domain(case):
    D = rt.DominoTiler
    if case.get("domain") == "rectangle":
        return D.Rectangle(case["rows"], case["cols"])
    return D.AztecDiamond(case["order"] if "order" in case else case["rows"])


def _bibone_start(case):
    T = rt.TriangleDimerTiler
    if case["domain"] == "rhombus":
        return T.RhombusBrick(case["rows"], case["cols"])
    return T.IceCreamCone(case["rows"], case["cols"])


def _q(case):
    return case["q"] or None


def _batch_jobs(case, r):
    """Half diamonds (every other one two-periodic), half hexagons, sizes uniform (the same for
    every seed: the seed gives the instances' randomness and weights)."""
    start, jobs, sizes = {}, [], random.Random(20261203)
    for k in range(case["count"]):
        model = "domino" if k % 2 == 0 else "lozenge"
        lo, hi = (case["order_lo"], case["order_hi"]) if model == "domino" else (case["side_lo"], case["side_hi"])
        size = sizes.randint(lo, hi)
        if (model, size) not in start:
            T = rt.DominoTiler if model == "domino" else rt.LozengeTiler
            d = T.AztecDiamond(size) if model == "domino" else T.Hexagon(size)
            start[model, size] = T.MaxTiling(d), T.MinTiling(d)
        tmax, tmin = start[model, size]
        weighted = model == "domino" and k % 4 == 2
        jobs.append({"model": model, "tmax": tmax, "tmin": tmin, "seed": r.getrandbits(31), "stream": k,
                     "rule": "cftp_twoperiodic" if weighted else "cftp", "a": 1.0,
                     "b": r.uniform(case["b_lo"], 1.0) if weighted else 1.0, "first_steps": 16, "max_attempts": 16})
    return jobs


def prepare(case, seed):
    rt.tune_load(TUNE_TABLE)
    r = random.Random(seed)
    s = {"case": case, "seed": r.getrandbits(31)}
    kind = case["kind"]
    if kind == "domino_walk":
        s["start"] = rt.DominoTiler.MinTiling(_domino_domain(case))
        s["tiler"] = rt.DominoTiler(rule=case["rule"], rng=case["rng"], a=case["a"], b=case["b"])
        if case["table"]:  # one parameter set per generator, as LoadTinyMT of a parameter file gives
            n = rt.side_of(s["start"])
            s["tiler"].LoadTinyMT(np.random.RandomState(seed & 0x7FFFFFFF).randint(
                0, 2**32, size=((n - 2) * (n // 2 - 2), 3), dtype=np.uint32))
    elif kind == "domino_coupled":
        d = _domino_domain(case)
        tmax, tmin = rt.DominoTiler.MaxTiling(d), rt.DominoTiler.MinTiling(d)
        n = rt.side_of(tmax)
        s["tiler"] = rt.DominoTiler(rule="cftp_twoperiodic", rng=case["rng"], a=case["a"], b=case["b"])
        s["chains"] = c = rt.DominoSampler(n, 4, s["tiler"])
        for k, t in enumerate((tmin, tmax, tmin, tmax)):  # 0, 1 are swept, 2, 3 keep the start
            c.load(k, t)
        c.set_active(2)
        c.set_domain(d)
        c.sync()
        s["colours"] = rt.mt19937_colours(s["seed"], case["steps"])
        s["heights"] = [torch.empty(n * n, dtype=torch.int32, device="cuda") for _ in range(2)]
    elif kind == "domino_cftp":
        d = _domino_domain(case)
        s["max"], s["min"] = rt.DominoTiler.MaxTiling(d), rt.DominoTiler.MinTiling(d)
        s["tiler"] = rt.DominoTiler(rule=case["rule"], rng=case["rng"], a=case["a"], b=case["b"])
    elif kind in ("lozenge_walk", "lozenge_cftp"):
        d = rt.LozengeTiler.Hexagon(case["side"])
        s["max"], s["start"] = rt.LozengeTiler.MaxTiling(d), rt.LozengeTiler.MinTiling(d)
        s["tiler"] = rt.LozengeTiler(rng=case["rng"], q=_q(case))
    elif kind == "recttri_walk":
        s["start"] = rt.RectTriangleTiler.minHex(case["side"])
        w = [round(r.uniform(0.7, 1.4), 3) for _ in range(9)] if case["weighted"] else None
        s["tiler"] = rt.RectTriangleTiler(rng=case["rng"], weights=w)
    elif kind == "bibone_walk":
        s["start"] = _bibone_start(case)
        s["tiler"] = rt.TriangleDimerTiler(rng=case["rng"])
    elif kind in ("six_walk", "six_cftp"):
        T = rt.SixVertexTiler
        s["start"], s["max"] = T.MinHeight(case["n"]), T.MaxHeight(case["n"])
        s["tiler"] = T(case["a"], case["b"], case["c"])
    else:
        s["jobs"] = _batch_jobs(case, r)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "domino_coupled":
        c = s["chains"]
        c.copy_chain(0, 2)
        c.copy_chain(1, 3)
        if case["rng"] == "tinymt":
            c.seed(s["seed"])
            c.run(s["colours"])
        else:
            c.run_fast(s["seed"], -case["steps"], case["steps"])
        for k in range(2):
            c.accumulate_heights(k, 0, s["heights"][k].data_ptr())
        return {"apart": c.diff(0, 1), "heights": s["heights"]}
    if kind == "domino_cftp":
        t, st = s["tiler"].cftp(s["max"], s["min"], s["seed"], first_steps=case["first"], schedule=1, max_attempts=16)
        return {"sample": t, "look_back": st["final_steps"]}
    if kind == "lozenge_cftp":
        t, st = s["tiler"].cftp(s["max"], s["start"], s["seed"], first_steps=case["first"], schedule=1, max_attempts=16)
        return {"sample": t, "look_back": st["final_steps"]}
    if kind == "six_cftp":
        t, st = s["tiler"].cftp(s["max"], s["start"], s["seed"], first_sweeps=case["first"], max_attempts=16)
        return {"sample": t, "look_back": st["final_steps"]}
    if kind == "batch":
        samples, attempts, _ = rt.cftp_batch(s["jobs"])
        return {"samples": np.concatenate(samples), "attempts": np.array(attempts)}
    t = s["start"].copy()  # Walk changes the caller's tiling
    s["tiler"].Walk(t, case["sweeps"] if kind == "six_walk" else case["steps"], s["seed"])
    return t


# Integer operations of one flip attempt: the draw (TinyMT32: about 16; a quarter of a
# Philox4x32-10 block: about 20; a bit-sliced heat bath: about 8 of a 32-point word's 256) and
# the decision.
_OPS = {"tinymt": 20, "fast": 24}


def work(case):
    """Bytes: the start state(s) read and the result written once (int32).  Operations: the
    flip attempts of the pass, at the look-back that such sizes need where it is random."""
    kind = case["kind"]
    if kind == "domino_walk":
        area = case["rows"] * case["cols"] * (2 if case["domain"] == "aztec" else 1)
        n = 2 * case["rows"] + 6 if case["domain"] == "aztec" else max(case["rows"], case["cols"]) + 5
        return {"bytes": 8 * n * n, "flops": area / 2 * case["steps"] * _OPS[case["rng"]]}
    if kind == "domino_coupled":
        n = 2 * case["order"] + 6
        return {"bytes": 2 * n * n + 8 * n * n, "flops": 2 * case["order"] ** 2 * case["steps"] * _OPS[case["rng"]]}
    if kind == "domino_cftp":
        o = case["order"]  # look-back of about 8 order^2 half-sweeps, doubled: twice that in all
        return {"bytes": 12 * (2 * o + 6) ** 2, "flops": 2 * o * o * 16 * o * o * _OPS[case["rng"]]}
    if kind in ("lozenge_walk", "lozenge_cftp"):
        n = case["side"]
        steps = case["steps"] if kind == "lozenge_walk" else 2 * 12 * n * n
        chains = 1 if kind == "lozenge_walk" else 2
        return {"bytes": 4 * (chains + 1) * (2 * n + 7) ** 2, "flops": chains * n * n * steps * _OPS[case["rng"]]}
    if kind == "recttri_walk":
        n = case["side"]
        return {"bytes": 8 * (2 * n + 7) ** 2, "flops": n * n * case["steps"] * _OPS[case["rng"]]}
    if kind == "bibone_walk":
        sites = case["rows"] * case["cols"] if case["domain"] == "rhombus" else case["rows"] ** 2 / 2
        side = 2 * (max(case["rows"], case["cols"]) + 6)
        return {"bytes": 8 * side * side, "flops": sites / 3 * case["steps"] * _OPS[case["rng"]]}
    if kind in ("six_walk", "six_cftp"):
        n = case["n"]
        sweeps = case["sweeps"] if kind == "six_walk" else 2 * 2 * n * n
        chains = 1 if kind == "six_walk" else 2
        return {"bytes": 4 * (chains + 1) * (n + 1) ** 2, "flops": chains * n * n * sweeps * 8}
    o, h = (case["order_lo"] + case["order_hi"]) / 2, (case["side_lo"] + case["side_hi"]) / 2
    per = 2 * o * o * 16 * o * o + 2 * h * h * 24 * h * h
    return {"bytes": case["count"] / 2 * 12 * ((2 * o + 6) ** 2 + (2 * h + 7) ** 2), "flops": case["count"] / 2 * per * 24}
