"""Post-processing sums at the edges of their kernels, bit for bit against the oracle: slots that end inside a warp,
one class and thirty-two, a class without grains, a domain whose only snapshot is its last, domains that end at
different times."""
import numpy as np
import pytest

import oracle
import score_gb300 as sg

pytestmark = pytest.mark.gpu

BOXES = [((24, 24, 24), 17, 6, ["0.0", "0.5", "0.9"]), ((33, 20, 27), 40, 33, ["0.95"]), ((20, 41, 22), 9, 12, ["0.1", "0.2", "0.3", "0.4"])]


@pytest.fixture(scope="module")
def ensemble(tmp_path_factory):
    td = tmp_path_factory.mktemp("post")
    params, doms = [], []
    for k, ((nx, ny, nz), ng, nn, logs) in enumerate(BOXES):
        params.append(sg.read_uds(sg.UdsSpec(nx=nx, ny=ny, nz=nz, logpoints=logs, border_policy=1).write(td / f"{k}.uds")))
        doms.append(sg.generate_domain(nx, ny, nz, ng, nn, seed=70 + k))
    with sg.Batch(params) as b:
        for k, d in enumerate(doms):
            b.load_domain(k, d)
        b.place_nuclei()
        b.run_until()
        evo = []
        for k, d in enumerate(doms):
            log = b.grainevo(k)
            rx, deformed = b.grain_counts(k)
            evo.append({"ndefg": d.ndefg, "nrxg": d.nrxg, "t": np.array([x[0].t for x in log]), "counts": np.array([x[1] for x in log]),
                        "final": np.concatenate([deformed, rx]), "tsimend": b.stats(k).t, "cells": d.ncells})
        yield b, doms, evo


@pytest.mark.parametrize("nslots", [2, 31, 32, 33, 257])
def test_kinetics(gpu, ensemble, nslots):
    b, _, evo = ensemble
    t, v, box = b.rediscr_kinetics(nslots)
    t0, v0, box0 = oracle.rediscr_kinetics(evo, nslots)
    assert np.array_equal(t, t0) and np.array_equal(v, v0) and box == box0


@pytest.mark.parametrize("nclass,skip", [(1, None), (2, 0), (5, 3), (32, 31)])
@pytest.mark.parametrize("nslots", [2, 65])
def test_texture(gpu, ensemble, nclass, skip, nslots):
    b, doms, evo = ensemble
    n = sum(d.ndefg + d.nrxg for d in doms)
    cls = np.random.default_rng(nclass).integers(0, nclass, size=n).astype(np.uint32)
    if skip is not None:
        cls[cls == skip] = (skip + 1) % nclass
    off = np.cumsum([0] + [d.ndefg + d.nrxg for d in doms])
    for k, e in enumerate(evo):
        e["cls"] = cls[off[k]:off[k + 1]]
    t, v = b.rediscr_texture(nslots, cls, nclass)
    t0, v0 = oracle.rediscr_texture(evo, nslots, nclass)
    assert np.array_equal(t, t0) and np.array_equal(v, v0)
