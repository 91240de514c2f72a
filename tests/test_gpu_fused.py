"""Growth steps inside one launch (small fronts) against the oracle, and against the separate kernels.

The fused path takes over by front size, so the cases sit at its edges: a front of less than one tile, one
just past a tile, both lists, every grow mode (dt changes, refresh from the weights and from the cached
mobilities, nuclei and defragmentation between launches), one step a call, a group of one block, and more
full cells in a block than its shared records hold.  FP64 results are the oracle's bits; FP32 results are
the separate kernels' bits.
"""
import numpy as np
import pytest

import oracle
import score_gb300 as sg
from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu

RECOVERY = {"recovery": 10}
HEATING = {"schedule": [("0.0", "700.0"), ("0.05", "760.0"), ("360000.0", "760.0")]}
# (box, grains, nuclei, generator and parameter overrides)
CASES = {
    "one_nucleus": ((17, 19, 23), 3, 1, {}, {}),
    "one_tile": ((24, 24, 24), 8, 6, {}, {}),
    "odd_periodic": ((45, 33, 51), 40, 30, {}, {"boundary": 1, "border_policy": 1}),
    "thin": ((96, 5, 64), 12, 20, {}, {"border_policy": 1}),
    "heating": ((50, 44, 40), 25, 16, {}, HEATING),
    "heating_rh": ((50, 44, 40), 25, 16, {}, {**HEATING, "mobility_model": 2}),
    "recovery_nuclei": ((60, 50, 40), 30, 60, {"nucleation_rate": 400.0}, RECOVERY),
    "recovery_mp": ((50, 50, 50), 25, 16, {}, {"recovery": 3}),
    "defrag": ((52, 50, 48), 25, 16, {}, {"defragmentation": 1, "defrag_x": ["0.2", "0.5", "0.8"]}),
    "many_full": ((64, 64, 64), 1, 2500, {}, {"border_policy": 1}),
}


def make(name, tmp_path, **kw):
    (nx, ny, nz), ng, nn, gen, par = CASES[name]
    d = sg.generate_domain(nx, ny, nz, ng, nn, seed=31, **gen)
    return sg.read_uds(sg.UdsSpec(nx=nx, ny=ny, nz=nz, **{**par, **kw}).write(tmp_path / f"{name}.uds")), d


@pytest.mark.parametrize("use_graph", [1, 0])
@pytest.mark.parametrize("name", sorted(CASES))
def test_fused_steps_match_oracle(gpu, tmp_path, name, use_graph):
    """use_graph 0 keeps the separate kernels: both give the oracle's bits."""
    p, d = make(name, tmp_path)
    ref = oracle.run(p, d)
    assert ref["status"] == 0
    with sg.GrowthMachine(p) as gm:
        gm.set_tune(use_graph=use_graph)
        gm.load_domain(d)
        gm.place_nuclei()
        n0 = gm.timing().kernel_launches
        tr = gm.run_until()
        if use_graph:
            assert gm.timing().kernel_launches - n0 < 5 * len(tr), "the separate kernels ran"
        assert_same(tr, gm.labels(), *gm.grain_counts(), ref)


@pytest.mark.parametrize("name", ["odd_periodic", "heating", "recovery_nuclei", "defrag"])
def test_one_step_a_call_and_mixed_paths(gpu, tmp_path, name):
    """score_step, and a run that changes between the two paths on the way, give the same steps."""
    p, d = make(name, tmp_path)
    ref = oracle.run(p, d)
    with sg.GrowthMachine(p) as gm:
        gm.load_domain(d)
        gm.place_nuclei()
        tr = []
        for k in range(len(ref["trace"])):
            gm.set_tune(use_graph=0 if k % 7 in (2, 3) else 1)
            tr.append(gm.step())
        assert_same(tr, gm.labels(), *gm.grain_counts(), ref)
        gm.restart()
        gm.place_nuclei()
        gm.set_tune(use_graph=1)
        tr = [gm.step() for _ in range(5)] + gm.run_until()
        assert_same(tr, gm.labels(), *gm.grain_counts(), ref)


@pytest.mark.parametrize("name", ["one_tile", "odd_periodic", "heating_rh", "recovery_nuclei", "many_full"])
def test_fp32_fused_equals_separate_kernels(gpu, tmp_path, name):
    p, d = make(name, tmp_path, precision=1)
    out = []
    for use_graph in (1, 0):
        with sg.GrowthMachine(p) as gm:
            gm.set_tune(use_graph=use_graph)
            gm.load_domain(d)
            gm.place_nuclei()
            tr = gm.run_until()
            out.append((np.array([(s.t, s.Xcells, s.Sv, s.Pmax, s.n_new) for s in tr]), gm.labels()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("ndom", [2, 48])
def test_batch_groups(gpu, tmp_path, ndom):
    """Groups of many blocks and of few (tiles by the dozen a block, more full cells than a block's shared
    records hold), stopped by max_steps on the way."""
    names = ["many_full", "one_nucleus", "odd_periodic"]
    cases = [make(n, tmp_path) for n in names]
    refs = [oracle.run(p, d) for p, d in cases]
    pick = [0 if i % 3 != 1 else 1 + (i // 3) % 2 for i in range(ndom)]
    with sg.Batch([cases[k][0] for k in pick]) as b:
        for i, k in enumerate(pick):
            b.load_domain(i, cases[k][1])
        b.place_nuclei()
        assert b.run_until(max_steps=9) == 9
        first = [b.trace(i) for i in range(ndom)]
        b.run_until()
        for i, k in enumerate(pick):
            assert_same(first[i] + b.trace(i), b.labels(i), *b.grain_counts(i), refs[k])


def test_contexts_one_after_another(gpu, tmp_path):
    """A new context's mailbox may be the pinned memory of one that has gone: nothing in it counts."""
    short, long = make("one_tile", tmp_path), make("odd_periodic", tmp_path)
    refs = [oracle.run(p, d) for p, d in (short, long)]
    assert len(refs[0]["trace"]) < len(refs[1]["trace"])
    for _ in range(3):
        for (p, d), ref in zip((short, long), refs):
            with sg.GrowthMachine(p) as gm:
                gm.load_domain(d)
                gm.place_nuclei()
                tr = gm.run_until()
                assert_same(tr, gm.labels(), *gm.grain_counts(), ref)
        pick = [short, long, short, long]
        with sg.Batch([p for p, _ in pick]) as b:
            for i, (_, d) in enumerate(pick):
                b.load_domain(i, d)
            b.place_nuclei()
            b.run_until()
            for i in range(4):
                assert_same(b.trace(i), b.labels(i), *b.grain_counts(i), refs[i % 2])
