"""The work that users of the growth library have it do, as cases whose speed and results can be measured.

Kinds of case:

  grow         one domain through ``GrowthMachine``: the structure comes from pinned host buffers, the
               nuclei are placed, the domain is stepped until X > 0.99 and the labels and per-grain cell
               counts go back to the host (the sequence of the growth machine's caller)
  batch        an ensemble of uneven independent domains through ``Batch``, the same sequence
  percolation  cluster analysis of a partly recrystallized domain
  postprocess  rediscretized kinetics, macrotexture and grain sizes over an ensemble's grain-evolution logs
  synthesis    the deformed structure, orientations, densities and nuclei of a new domain
  weights      the table of mobility weights P(rx grain, deformed grain) on the device
"""
from __future__ import annotations

import ctypes as C
import math
import random
import tempfile
from pathlib import Path

import numpy as np
import torch

import score_gb300 as sg
from score_gb300 import growth as sg_growth

X_TARGET = 0.99
# the benchmark domains' densities: a 512^3 domain holds 20,000 deformed grains and 50,000 nuclei,
# a 128^3 one 500 grains and 200 nuclei
CELLS_PER_GRAIN_512, CELLS_PER_NUCLEUS_512 = 512 ** 3 / 20000, 512 ** 3 / 50000
CELLS_PER_GRAIN_128, CELLS_PER_NUCLEUS_128 = 128 ** 3 / 500, 128 ** 3 / 200
LOGPOINTS = ["0.0", "0.1", "0.2", "0.3", "0.4", "0.5", "0.6", "0.7", "0.8", "0.9"]
# rolled structure: flat grains 1:4:8, three texture components, two stored energies, nuclei at boundaries
PANCAKE = dict(aspect=(1.0, 4.0, 8.0), ori_mode=1, ncomp=3, scatter_deg=10.0, rho_mode=1, rho_lo=1e14, rho_hi=5e15,
               site_mode=1, gb_fraction=0.8)
RH = (0.9, 5.0, 9.0)  # the Rollett-Holm sigmoid's cut, transition and exponent
GROW = {"kind": "grow", "precision": 0, "pancake": False, "recovery": False, "rate": 0.0, "heating": False, "mobility": 1,
        "boundary": 0, "grow_border": False, "stepwise": False}


def listed():
    return [
        # a small structure stepped one call at a time, as a program does that couples the growth to
        # something of its own: launches and waits count
        {**GROW, "name": "grow_64_fp64", "nx": 64, "ny": 64, "nz": 64, "grains": 40, "nuclei": 24, "stepwise": True},
        # the standard small study
        {**GROW, "name": "grow_128_fp64", "nx": 128, "ny": 128, "nz": 128, "grains": 500, "nuclei": 200},
        # an uneven box cut from a map, heated while it grows (every mobility moves on every step),
        # Rollett-Holm mobilities, periodic in z too, FP32 + Kahan fill
        {**GROW, "name": "grow_odd_heated_fp32", "nx": 171, "ny": 93, "nz": 139, "grains": 331, "nuclei": 405, "precision": 1,
         "heating": True, "mobility": 2, "boundary": 1, "grow_border": True},
        # the benchmark domain
        {**GROW, "name": "grow_512_fp64", "nx": 512, "ny": 512, "nz": 512, "grains": 20000, "nuclei": 50000},
        # recovering deformed grains (every driving force moves on every step) and nuclei that appear
        # during the run
        {**GROW, "name": "grow_384_recovery_fp32", "nx": 384, "ny": 384, "nz": 384, "grains": 8438, "nuclei": 21094, "precision": 1,
         "recovery": True, "rate": 422.0},
        # rolled sheet
        {**GROW, "name": "grow_384_pancake_fp64", "nx": 384, "ny": 384, "nz": 384, "grains": 422, "nuclei": 10547, "pancake": True},
        # ensembles of solitary units: edges 64 to 256, 100 to 5,000 grains, 50 to 2,000 nuclei
        {"name": "batch_16_fp32", "kind": "batch", "domains": 16, "lo": 64, "hi": 256, "shapes": 1, "precision": 1, "logged": False},
        # the same with the grain-evolution log at ten recrystallized fractions
        {"name": "batch_12_logged_fp64", "kind": "batch", "domains": 12, "lo": 64, "hi": 192, "shapes": 2, "precision": 0, "logged": True},
        # which rx clusters span the sample, with every cell's cluster
        {"name": "percolation_256", "kind": "percolation", "nx": 256, "ny": 256, "nz": 256, "grains": 2500, "nuclei": 6250, "x": 0.15,
         "connected": False},
        # the averages over an ensemble, on the 1,000 times of RediscretizationSteps
        {"name": "postprocess_12", "kind": "postprocess", "domains": 12, "lo": 64, "hi": 128, "shapes": 3, "slots": 1000, "classes": 8},
        # a new structure
        {"name": "synthesis_256", "kind": "synthesis", "nx": 256, "ny": 256, "nz": 256, "grains": 2500, "nuclei": 6250, "pancake": False},
        # every weight of a domain's pools
        {"name": "weights_2000x1500", "kind": "weights", "nrxg": 2000, "ndefg": 1500, "mobility": 1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo_cells, hi_cells, least):
    """Three uneven edges whose product is about log-uniform in [lo_cells, hi_cells]."""
    edge = math.exp(rng.uniform(math.log(lo_cells), math.log(hi_cells))) ** (1 / 3)
    a, b = math.exp(rng.uniform(-0.35, 0.35)), math.exp(rng.uniform(-0.35, 0.35))
    return {"nx": max(least, round(edge * a)), "ny": max(least, round(edge * b)), "nz": max(least, round(edge / (a * b)))}


def _pools(rng, box):
    """Grain and nucleus counts between the two benchmark domains' densities."""
    n, f, g = box["nx"] * box["ny"] * box["nz"], rng.random(), rng.random()
    return {"grains": max(8, round(n / (CELLS_PER_GRAIN_128 ** f * CELLS_PER_GRAIN_512 ** (1 - f)))),
            "nuclei": max(8, round(n / (CELLS_PER_NUCLEUS_128 ** g * CELLS_PER_NUCLEUS_512 ** (1 - g))))}


def draw(rng):
    kind = rng.choice(["grow", "grow", "grow", "batch", "percolation", "postprocess", "synthesis", "weights"])
    if kind == "grow":
        box = _box(rng, 48 ** 3, 320 ** 3, 40)
        recovery = rng.random() < 0.2
        c = {**GROW, **box, **_pools(rng, box), "precision": rng.randrange(2), "recovery": recovery,
             "heating": not recovery and rng.random() < 0.2, "pancake": rng.random() < 0.25, "mobility": 2 if rng.random() < 0.25 else 1,
             "boundary": rng.randrange(2), "grow_border": True, "stepwise": rng.random() < 0.25}
        if recovery:
            c["rate"] = float(max(20, round(1000 * box["nx"] * box["ny"] * box["nz"] / 512 ** 3)))
        return c
    if kind == "batch":
        lo = _log_int(rng, 48, 80)
        return {"kind": "batch", "domains": _log_int(rng, 2, 16), "lo": lo, "hi": _log_int(rng, lo + 10, 224),
                "shapes": rng.randrange(1 << 20), "precision": rng.randrange(2), "logged": rng.random() < 0.3}
    if kind == "percolation":
        box = _box(rng, 50 ** 3, 280 ** 3, 40)
        return {"kind": "percolation", **box, **_pools(rng, box), "x": round(rng.uniform(0.02, 0.9), 3), "connected": rng.random() < 0.5}
    if kind == "postprocess":
        return {"kind": "postprocess", "domains": _log_int(rng, 1, 14), "lo": 56, "hi": _log_int(rng, 66, 128),
                "shapes": rng.randrange(1 << 20), "slots": _log_int(rng, 100, 1500), "classes": rng.randint(1, 32)}
    if kind == "synthesis":
        box = _box(rng, 48 ** 3, 280 ** 3, 24)
        return {"kind": "synthesis", **box, **_pools(rng, box), "pancake": rng.random() < 0.3}
    return {"kind": "weights", "nrxg": _log_int(rng, 20, 3000), "ndefg": _log_int(rng, 20, 1500), "mobility": 1 + rng.randrange(2)}


def _shapes(case):
    """(nx, ny, nz, grains, nuclei) of an ensemble's domains: edges, grains and nuclei as the benchmark's
    ensemble draws them, the pools no denser than a tenth of a per cent of the cells."""
    r = random.Random(case["shapes"])
    out = []
    for _ in range(case["domains"]):
        e = [r.randint(case["lo"], case["hi"]) for _ in range(3)]
        most = e[0] * e[1] * e[2] // 1000
        out.append((*e, min(r.randint(100, 5000), most), min(r.randint(50, 2000), most)))
    return out


def _params(nx, ny, nz, **kw):
    """Parameters by way of the input file that a user of the reference has."""
    with tempfile.TemporaryDirectory() as td:
        return sg.read_uds(sg.UdsSpec(nx=nx, ny=ny, nz=nz, **kw).write(Path(td) / "case.uds"))


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def _domain(nx, ny, nz, grains, nuclei, seed, pinned=True, **kw):
    d = sg.generate_domain(nx, ny, nz, grains, nuclei, seed=seed, device=0, **kw)
    if not pinned:
        return d
    return sg.Domain(nx, ny, nz, *(_pinned(x) for x in (d.grid, d.defg_quat, d.defg_rho0, d.rxg_quat, d.rxg_site, d.rxg_tincub)))


def _label_buffer(d):
    return torch.empty((d.nz, d.ny, d.nx), dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)


MOST_STEPS = 8192


def _trace(runs):
    """X(t) of runs and the front's work, one row a run, as a program keeps them to plot: rows end in zeros."""
    out = {"t": np.zeros((len(runs), MOST_STEPS)), "cells": np.zeros((len(runs), MOST_STEPS)),
           "front": np.zeros((len(runs), MOST_STEPS), dtype=np.int64)}
    for i, rows in enumerate(runs):
        rows = rows[:MOST_STEPS]
        out["t"][i, :len(rows)] = [s.t for s in rows]
        out["cells"][i, :len(rows)] = [s.Xcells for s in rows]
        out["front"][i, :len(rows)] = [s.Sv for s in rows]
    return out


def _grow_params(case):
    kw = {"precision": case["precision"], "boundary": case["boundary"], "border_policy": 1 if case["grow_border"] else 0,
          "mobility_model": case["mobility"]}
    if case["recovery"]:
        kw["recovery"] = 10
    if case["heating"]:
        kw["schedule"] = [("0.0", "700.0"), ("0.05", "760.0"), ("360000.0", "760.0")]
    return _params(case["nx"], case["ny"], case["nz"], **kw)


def _grown_batch(case, seed, logged, precision, grow):
    shapes = _shapes(case)
    kw = {"logpoints": LOGPOINTS} if logged else {}
    b = sg.Batch([_params(*s[:3], precision=precision, border_policy=1, **kw) for s in shapes])
    doms = [_domain(*s, seed=seed * 1000 + i) for i, s in enumerate(shapes)]
    for i, d in enumerate(doms):
        b.load_domain(i, d)
    if grow:
        b.place_nuclei()
        b.run_until(X_TARGET)
    return b, doms


def prepare(case, seed):
    kind = case["kind"]
    if kind == "grow":
        kw = dict(PANCAKE) if case["pancake"] else {}
        if case["rate"]:
            kw["nucleation_rate"] = case["rate"]
        d = _domain(case["nx"], case["ny"], case["nz"], case["grains"], case["nuclei"], seed, **kw)
        gm = sg.GrowthMachine(_grow_params(case))
        gm.load_domain(d)
        return {"case": case, "gm": gm, "domain": d, "labels": _label_buffer(d)}
    if kind == "batch":
        b, doms = _grown_batch(case, seed, case["logged"], case["precision"], grow=False)
        return {"case": case, "batch": b, "domains": doms, "labels": [_label_buffer(d) for d in doms]}
    if kind == "percolation":
        d = _domain(case["nx"], case["ny"], case["nz"], case["grains"], case["nuclei"], seed, pinned=False)
        gm = sg.GrowthMachine(_params(case["nx"], case["ny"], case["nz"], border_policy=1))
        gm.load_domain(d)
        gm.place_nuclei()
        gm.run_until(case["x"])
        return {"case": case, "gm": gm}
    if kind == "postprocess":
        b, doms = _grown_batch(case, seed, True, 0, grow=True)
        n = sum(d.ndefg + d.nrxg for d in doms)
        cls = np.random.default_rng(seed).integers(0, case["classes"], size=n).astype(np.uint32)
        return {"case": case, "batch": b, "classes": cls}
    if kind == "synthesis":
        return {"case": case, "seed": seed, "kw": dict(PANCAKE) if case["pancake"] else {}}
    qr, qd = _orientations(case, seed)
    p = sg.default_params()
    p.mobility_model = case["mobility"]
    p.RH_cut, p.RH_trans, p.RH_exponent = RH
    dev = torch.device("cuda:0")
    return {"case": case, "params": p, "qr": torch.from_numpy(qr).to(dev), "qd": torch.from_numpy(qd).to(dev),
            "table": torch.empty((case["nrxg"], case["ndefg"]), dtype=torch.float64, device=dev),
            "pmax": torch.empty(1, dtype=torch.float64, device=dev)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "grow":
        gm = state["gm"]
        gm.load_domain(state["domain"])
        gm.place_nuclei()
        if case["stepwise"]:
            rows = []
            while not rows or rows[-1].X <= X_TARGET:
                rows.append(gm.step())
        else:
            rows = gm.run_until(X_TARGET)
        labels = gm.labels(state["labels"])
        rx, deformed = gm.grain_counts()
        return {**_trace([rows]), "labels": labels.view(np.int32), "rx": rx.view(np.int32), "deformed": deformed.view(np.int32)}
    if kind == "batch":
        b = state["batch"]
        for i, d in enumerate(state["domains"]):
            b.load_domain(i, d)
        b.place_nuclei()
        b.run_until(X_TARGET)
        n = len(state["domains"])
        out = {"labels": [b.labels(i, state["labels"][i]).view(np.int32) for i in range(n)],
               "trace": _trace([b.trace(i) for i in range(n)]),
               "sizes": b.final_grain_sizes().view(np.int32)}
        if case["logged"]:
            logs = [x for i in range(n) for x in b.grainevo(i)]
            out["log"] = {"t": np.array([x[0].t for x in logs]), "counts": np.concatenate([x[1] for x in logs]).view(np.int32),
                          "area": np.concatenate([x[2].reshape(-1) for x in logs]).view(np.int32)}
        return out
    if kind == "percolation":
        r = state["gm"].percolation(connected=case["connected"], labels=True)
        sizes = np.zeros(1 << 16, dtype=np.int32)  # the largest clusters, ascending
        sizes[max(0, sizes.size - r["sizes"].size):] = r["sizes"][-sizes.size:]
        return {"labels": r["labels"].view(np.int32), "sizes": sizes, "PL": r["PL"],
                "clusters": int(r["n_clusters"]), "largest": int(r["largest"]), "spans": int(r["spans"])}
    if kind == "postprocess":
        b = state["batch"]
        t, v, box = b.rediscr_kinetics(case["slots"])
        t2, tex = b.rediscr_texture(case["slots"], state["classes"], case["classes"])
        return {"t": t, "rx": v, "box": box, "t2": t2, "texture": tex, "sizes": b.final_grain_sizes().view(np.int32)}
    if kind == "synthesis":
        d = sg.generate_domain(case["nx"], case["ny"], case["nz"], case["grains"], case["nuclei"], seed=state["seed"], device=0,
                               **state["kw"])
        return {"grid": d.grid.view(np.int32), "defg_quat": d.defg_quat, "rho": d.defg_rho0, "rxg_quat": d.rxg_quat,
                "site": d.rxg_site.view(np.int32), "tincub": d.rxg_tincub}
    qr, qd = state["qr"], state["qd"]
    rc = sg_growth.lib().score_mobility_table_noalloc(C.byref(state["params"]), qr.data_ptr(), qr.shape[0], qd.data_ptr(), qd.shape[0],
                                                      state["table"].data_ptr(), state["pmax"].data_ptr(),
                                                      C.c_void_p(torch.cuda.current_stream().cuda_stream))
    if rc != 0:
        raise RuntimeError(f"mobility table: status {rc}")
    return {"table": state["table"], "pmax": state["pmax"]}


def work(case):
    """Bytes and operations that the path cannot do without.

    Growth: the structure is read once and the labels written once; a cell stays in the front for about 44
    steps in the benchmark domain (30 to 45 in the small ones), and each of those updates reads its
    infector byte, increment and fill and writes the fill (FP64: 25 bytes and one addition; FP32 + Kahan:
    velocity, fill and compensation, 21 bytes and four); an infection attempt looks at 26 neighbours, once."""
    kind = case["kind"]
    if kind in ("grow", "batch"):
        boxes = [s[:3] for s in _shapes(case)] if kind == "batch" else [(case["nx"], case["ny"], case["nz"])]
        n = sum(x * y * z for x, y, z in boxes)
        updates = 40.0 * n
        return {"bytes": 8.0 * n + 26 * 4.0 * n + updates * (21 if case["precision"] else 25),
                "flops": updates * (4 if case["precision"] else 1)}
    if kind == "percolation":  # the grid in, the labels out; three lower neighbours of each cell
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 8.0 * n, "flops": 3.0 * n}
    if kind == "postprocess":  # ten snapshots and the final counts in, five operations a grain and time, twice
        grains = sum(s[3] + s[4] for s in _shapes(case))
        return {"bytes": 11 * 4.0 * grains + 8.0 * case["slots"] * (case["classes"] + 3), "flops": 2 * 5.0 * grains * case["slots"]}
    if kind == "synthesis":  # the labels out; about 30 seeds near a cell, eight operations each
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 4.0 * n, "flops": 30 * 8.0 * n}
    n = case["nrxg"] * case["ndefg"]  # the table out; a quaternion product, 24 candidates, twice where no low angle
    return {"bytes": 8.0 * n + 32.0 * (case["nrxg"] + case["ndefg"]), "flops": 150.0 * n}


# ---------------------------------------------------------------- mobility weights in plain 64 bits
def _unit(q):
    return q / np.linalg.norm(q, axis=-1, keepdims=True)


def _product(a, b):
    a0, a1, a2, a3 = a.unbind(-1)
    b0, b1, b2, b3 = b.unbind(-1)
    return torch.stack([a0 * b0 - a1 * b1 - a2 * b2 - a3 * b3, a0 * b1 + a1 * b0 + a2 * b3 - a3 * b2,
                        a0 * b2 - a1 * b3 + a2 * b0 + a3 * b1, a0 * b3 + a1 * b2 - a2 * b1 + a3 * b0], dim=-1)


def _rotation(axis, deg):
    h = np.radians(deg) / 2.0
    return np.concatenate([np.cos(h)[:, None], np.sin(h)[:, None] * _unit(axis)], axis=-1)


def _orientations(case, seed):
    """Uniform deformed grains; a third of the rx grains a small rotation away from one of them, a third
    near 40 deg <111>, the rest uniform."""
    rng = np.random.default_rng(seed)
    nr, nd = case["nrxg"], case["ndefg"]
    qd, qr = _unit(rng.normal(size=(nd, 4))), _unit(rng.normal(size=(nr, 4)))
    k = nr // 3
    src = rng.integers(0, nd, size=2 * k)
    turn = np.concatenate([_rotation(rng.normal(size=(k, 3)), rng.uniform(1.0, 12.0, size=k)),
                           _rotation(np.ones((k, 3)) + rng.normal(scale=0.03, size=(k, 3)), 40.0 + rng.uniform(-4.0, 4.0, size=k))])
    if k:
        qr[:2 * k] = _product(torch.from_numpy(qd[src]), torch.from_numpy(turn)).numpy()
    return np.ascontiguousarray(_unit(qr)), np.ascontiguousarray(qd)


def _candidates(p, q):
    """The 24 cubic equivalents of the misorientation q^-1 p as six quaternions, (..., 6, 4)."""
    r = _product(q * torch.tensor([1.0, -1.0, -1.0, -1.0], dtype=q.dtype, device=q.device), p)
    a, b, c, d = r.unbind(-1)
    f = math.sqrt(0.5)
    return torch.stack([torch.stack([(a + b) * f, (a - b) * f, (c + d) * f, (c - d) * f], -1),
                        torch.stack([(a + c) * f, (a - c) * f, (b + d) * f, (b - d) * f], -1),
                        torch.stack([(a + d) * f, (a - d) * f, (b + c) * f, (b - c) * f], -1),
                        torch.stack([a + b + c + d, a + b - c - d, a - b + c - d, a - b - c + d], -1) * 0.5,
                        torch.stack([a + b + c - d, a + b - c + d, a - b + c + d, a - b - c - d], -1) * 0.5, r], dim=-2)


def exact(case, seed):
    """The weights in 64 bits: -1 up to 15 degrees, cos^2 within 10 degrees of 40 deg <111>, else 0; or the
    sigmoid.  The other kinds give counts and labels, or are fixed by them (a growth run's times by its
    whole sequence of cell infections, the ensemble averages by the logs of such runs)."""
    if case["kind"] != "weights":
        return None
    qr, qd = (torch.from_numpy(x) for x in _orientations(case, seed))
    lagb = math.radians(15.0)
    h = math.radians(20.0)
    m40 = torch.tensor([math.cos(h)] + [math.sin(h) / math.sqrt(3.0)] * 3, dtype=torch.float64)
    rows = []
    for i in range(0, len(qr), 64):
        c = _candidates(qr[i:i + 64, None, :], qd[None, :, :])
        best, at = c.abs().amax(-1).max(-1)
        theta = 2.0 * torch.acos(best.clamp(max=1.0))
        if case["mobility"] == 2:
            rows.append(1.0 - RH[0] * torch.exp(-RH[1] * (theta / lagb) ** RH[2]))
            continue
        dis = torch.gather(c, 2, at[..., None, None].expand(*at.shape, 1, 4))[..., 0, :].abs().sort(dim=-1, descending=True).values
        dev = 2.0 * torch.acos(_candidates(dis, m40.expand_as(dis)).abs().amax((-1, -2)).clamp(max=1.0))
        w = torch.where(dev < math.radians(10.0), torch.cos(0.5 * math.pi * dev / math.radians(10.0)) ** 2, torch.zeros_like(dev))
        rows.append(torch.where(theta <= lagb, torch.full_like(w, -1.0), w))
    t = torch.cat(rows)
    return {"table": t, "pmax": t.max().reshape(1)}
