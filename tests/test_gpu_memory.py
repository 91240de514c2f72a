"""Device memory of a loaded domain and of post-processing: no list or workspace beyond what the domain's arrays take."""
import numpy as np
import pytest

import oracle
import score_gb300 as sg
from _limits import set_limits
from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


def used():
    import torch
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def test_loaded_domain(gpu, tmp_path):
    """192^3, FP64, 40 x 30 pairs: the arrays of the front, the grid, the masks and the request list; 24 MB for what a pool of
    2 MB pieces rounds up.  A list of weight-table entries must not follow the cells."""
    n = 192
    N = n**3
    d = sg.generate_domain(n, n, n, 40, 30, seed=3, device=0)
    p = sg.read_uds(sg.UdsSpec(nx=n, ny=n, nz=n).write(tmp_path / "p.uds"))
    with sg.GrowthMachine(p) as gm:  # kernels loaded, streams made
        gm.load_domain(d)
        gm.place_nuclei()
        gm.step()
    capB = 6 * n * n + 1
    front = 4 * 8 + 4 * 4 + 1          # fill, vel, inc, mob; grains, position, full list; infector
    masks = 2 / 8 + 2 * 8 * 4 / 1024   # full, INACTIVE; counts a tile of 1,024
    recycle = 4 * 0.1 * 0.1 * 10 * N   # at most: initial cache x fill a step x a factor below 10
    arrays = (front + masks) * (N + capB) + recycle + 6 * 4 * N + 8 * N
    with sg.GrowthMachine(p) as gm:
        before = used()
        gm.load_domain(d)
        assert used() - before <= arrays + 24 * 2**20


def test_restart_without_a_staging_buffer(gpu, tmp_path):
    """A restart that gets no buffer for the list of entries to clear (the refusal comes from a stand-in for the allocation)
    clears the whole table."""
    n = 48
    d = sg.generate_domain(n, n, n, 300, 1000, seed=5)
    d.rxg_tincub[12:] = 1e9  # 12 nuclei, a table of 300,000 pairs of which a run meets some hundreds
    p = sg.read_uds(sg.UdsSpec(nx=n, ny=n, nz=n, mobility_model=2, RH_exponent="1.0").write(tmp_path / "p.uds"))
    ref = oracle.run(p, d)
    with sg.GrowthMachine(p) as gm:
        gm.load_domain(d)
        gm.place_nuclei()
        tr = gm.run_until()
        assert 12 * 48 < 8 * sum(s.p_misses for s in tr) < 8 * 300 * 1000 / 64  # more than the nuclei's buffer, a listed restart
        set_limits(gm, stage=0)
        gm.restart()
        set_limits(gm)
        gm.place_nuclei()
        assert_same(gm.run_until(), gm.labels(), *gm.grain_counts(), ref)


def test_postprocessing_rows(gpu, tmp_path):
    """Six domains of 20,000 grains and up to 256 snapshots, some 400 MB of slopes: in groups, the sums the oracle's, and no
    large buffer kept after the call."""
    n = 48
    logs = [repr(round(0.0037 * k, 6)) for k in range(1, 257)]
    p = sg.read_uds(sg.UdsSpec(nx=n, ny=n, nz=n, logpoints=logs, border_policy=1).write(tmp_path / "p.uds"))
    doms = [sg.generate_domain(n, n, n, 20000, 24, seed=40 + k, device=0) for k in range(6)]
    with sg.Batch([p] * len(doms)) as b:
        for k, d in enumerate(doms):
            b.load_domain(k, d)
        b.place_nuclei()
        b.run_until()
        evo = []
        for k, d in enumerate(doms):
            log = b.grainevo(k)
            rx, deformed = b.grain_counts(k)
            evo.append({"ndefg": d.ndefg, "nrxg": d.nrxg, "t": np.array([x[0].t for x in log]), "counts": np.array([x[1] for x in log]),
                        "final": np.concatenate([deformed, rx]), "tsimend": b.stats(k).t, "cells": d.ncells,
                        "cls": (np.arange(d.ndefg + d.nrxg) % 3).astype(np.uint32)})
        assert sum((len(e["t"]) + 2) * e["ndefg"] * 16 for e in evo) > 300 * 2**20
        before = used()
        t, v, box = b.rediscr_kinetics(40)
        t2, v2 = b.rediscr_texture(40, np.concatenate([e["cls"] for e in evo]), 3)
        after = used()
        t0, v0, box0 = oracle.rediscr_kinetics(evo, 40)
        assert np.array_equal(t, t0) and np.array_equal(v, v0) and box == box0
        t0, v0 = oracle.rediscr_texture(evo, 40, 3)
        assert np.array_equal(t2, t0) and np.array_equal(v2, v0)
        assert after - before <= 72 * 2**20, "a large buffer was kept"
