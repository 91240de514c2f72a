"""Paths of the fused steps that small domains reach only with lower limits: four slots a thread, fronts that outgrow the
launch and its blocks on the way, and groups that leave before the host's answer (the next launch, or the separate
kernels, take the command again).  FP64: the oracle's bits; FP32: the separate kernels' bits.
"""
import numpy as np
import pytest

import oracle
import score_gb300 as sg
from score_gb300 import _abi
from _limits import set_limits
from test_gpu_fused import CASES, make
from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


def run(p, d, use_graph=1, **lim):
    """trace, labels, counts and launches of a run"""
    with sg.GrowthMachine(p) as gm:
        set_limits(gm, **lim)
        gm.set_tune(use_graph=use_graph)
        gm.load_domain(d)
        gm.place_nuclei()
        n0 = gm.timing().kernel_launches
        tr = gm.run_until()
        n = gm.timing().kernel_launches - n0
        return tr, gm.labels(), gm.grain_counts(), n


def as_array(tr):
    return np.array([(s.t, s.Xcells, s.Sv, s.Pmax, s.n_new) for s in tr])


@pytest.mark.parametrize("name", sorted(CASES))
def test_four_slots_a_thread(gpu, tmp_path, name):
    p, d = make(name, tmp_path)
    tr, labels, counts, n = run(p, d, wide=0)
    assert n < 5 * len(tr), "the separate kernels ran"
    assert_same(tr, labels, *counts, oracle.run(p, d))


@pytest.mark.parametrize("name", sorted(CASES))
def test_four_slots_a_thread_fp32(gpu, tmp_path, name):
    p, d = make(name, tmp_path, precision=1)
    tr, labels, counts, n = run(p, d, wide=0)
    assert n < 5 * len(tr), "the separate kernels ran"
    ref = run(p, d, use_graph=0)
    assert np.array_equal(as_array(tr), as_array(ref[0])) and np.array_equal(labels, ref[1])
    assert all(np.array_equal(a, b) for a, b in zip(counts, ref[2]))


@pytest.mark.parametrize("name", ["odd_periodic", "heating", "recovery_nuclei", "defrag"])
def test_front_outgrows_the_launch(gpu, tmp_path, name):
    """Fused below 3,000 slots, separate kernels above."""
    p, d = make(name, tmp_path)
    ref = oracle.run(p, d)
    tr, labels, counts, n = run(p, d, slots=3000)
    small = sum(sum(s.next_never) <= 3000 for s in tr)
    assert 0 < small < len(tr) - 5 and n > 5 * (len(tr) - small - 1)
    assert_same(tr, labels, *counts, ref)


def test_batch_outgrows_its_blocks(gpu, tmp_path):
    """16 slots a block of the launch: the batch goes on with the separate kernels."""
    names = ["odd_periodic", "one_nucleus", "heating", "recovery_nuclei"]
    cases = [make(n, tmp_path) for n in names]
    with sg.Batch([p for p, _ in cases]) as b:
        set_limits(b, block_slots=16)
        for i, (_, d) in enumerate(cases):
            b.load_domain(i, d)
        b.place_nuclei()
        steps = b.run_until()
        assert steps < b.timing().kernel_launches < 6 * steps, "one path only"
        for i, (p, d) in enumerate(cases):
            assert_same(b.trace(i), b.labels(i), *b.grain_counts(i), oracle.run(p, d))


# one poll is shorter than a round trip over the host link: nearly every group leaves, with the next command unread
@pytest.mark.parametrize("lim", [{}, {"slots": 3000}, {"wide": 0}], ids=["next_launch", "separate_kernels", "four_slots"])
@pytest.mark.parametrize("name", ["odd_periodic", "heating", "heating_rh", "recovery_nuclei", "recovery_mp", "defrag"])
def test_group_leaves_before_the_answer(gpu, tmp_path, name, lim):
    p, d = make(name, tmp_path)
    tr, labels, counts, n = run(p, d, host_polls=1, **lim)
    fused = sum(sum(s.next_never) <= lim.get("slots", 2**32) for s in tr)
    assert n >= fused // 2, "the groups stayed"
    assert_same(tr, labels, *counts, oracle.run(p, d))


def test_batch_leaves_before_the_answer(gpu, tmp_path):
    names = ["odd_periodic", "one_nucleus", "heating", "recovery_nuclei", "defrag", "many_full"]
    cases = [make(n, tmp_path) for n in names]
    for kw in ({"host_polls": 1}, {"host_polls": 1, "block_slots": 40}):
        with sg.Batch([p for p, _ in cases]) as b:
            set_limits(b, **kw)
            for i, (_, d) in enumerate(cases):
                b.load_domain(i, d)
            b.place_nuclei()
            b.run_until(max_steps=7)
            first = [b.trace(i) for i in range(len(names))]
            b.run_until()
            for i, (p, d) in enumerate(cases):
                assert_same(first[i] + b.trace(i), b.labels(i), *b.grain_counts(i), oracle.run(p, d))


@pytest.mark.parametrize("polls", [1, 4096])
def test_step_numbers_come_back(gpu, tmp_path, polls):
    """Numbers end at 2^24 - 1: the count passes its end in a run, in single calls, with groups that leave and without, and
    meets a number again after which a group once left."""
    last = 2**24 - 1
    p, d = make("recovery_nuclei", tmp_path)
    ref = oracle.run(p, d)
    assert len(ref["trace"]) > 60
    with sg.GrowthMachine(p) as gm:
        gm.load_domain(d)
        for first in (last - 40, last - 1, last, 1):
            set_limits(gm, number=first, host_polls=polls)
            gm.place_nuclei()
            tr = [gm.step() for _ in range(20)]
            set_limits(gm, host_polls=polls)
            tr += gm.run_until()
            assert_same(tr, gm.labels(), *gm.grain_counts(), ref)
            gm.restart()
        # every number of a run in which the groups left
        set_limits(gm, number=1000, host_polls=1)
        gm.place_nuclei()
        gm.run_until()
        gm.restart()
        set_limits(gm, number=1000)
        gm.place_nuclei()
        assert_same(gm.run_until(), gm.labels(), *gm.grain_counts(), ref)


def test_step_numbers_come_back_in_a_batch(gpu, tmp_path):
    names = ["odd_periodic", "heating", "many_full"]
    cases = [make(n, tmp_path) for n in names]
    with sg.Batch([p for p, _ in cases]) as b:
        set_limits(b, number=2**24 - 30)
        for i, (_, d) in enumerate(cases):
            b.load_domain(i, d)
        b.place_nuclei()
        b.run_until()
        for i, (p, d) in enumerate(cases):
            assert_same(b.trace(i), b.labels(i), *b.grain_counts(i), oracle.run(p, d))


@pytest.mark.parametrize("again", ["restart", "load"])
@pytest.mark.parametrize("name", ["odd_periodic", "recovery_nuclei"])
def test_restart_after_a_wait_gave_up(gpu, tmp_path, name, again):
    """One poll a wait: the group's first barrier gives up and the run ends with an error; a restart or a load puts the group's
    words back, and the next run is the oracle's."""
    p, d = make(name, tmp_path)
    ref = oracle.run(p, d)
    with sg.GrowthMachine(p) as gm:
        gm.load_domain(d)
        for _ in range(3):
            gm.place_nuclei()
            set_limits(gm, group_polls=1)
            with pytest.raises(sg.ScoreError) as e:
                gm.run_until()
            assert e.value.status == _abi.ERR_TIMEOUT
            with pytest.raises(sg.ScoreError):
                gm.run_until()
            set_limits(gm)
            gm.restart() if again == "restart" else gm.load_domain(d)
            gm.place_nuclei()
            assert_same(gm.run_until(), gm.labels(), *gm.grain_counts(), ref)
            gm.restart()


@pytest.mark.parametrize("at", [0, 1, 30])
@pytest.mark.parametrize("name", ["odd_periodic", "recovery_nuclei"])
def test_refused_launch(gpu, tmp_path, name, at):
    """A cooperative launch that is refused (the answer comes from a stand-in for the call): the separate kernels make the
    step, one call as well as a run, also the step of a command that its group did not read."""
    p, d = make(name, tmp_path)
    ref = oracle.run(p, d)
    n = len(ref["trace"])
    for singles, polls in ((n, 4096), (0, 4096), (0, 1)):
        with sg.GrowthMachine(p) as gm:
            set_limits(gm, refuse_after=at, host_polls=polls)
            gm.load_domain(d)
            gm.place_nuclei()
            tr = [gm.step() for _ in range(singles)]
            tr += gm.run_until()
            assert_same(tr, gm.labels(), *gm.grain_counts(), ref)


def test_stop_rules_wait_for_the_pending_step(gpu, tmp_path):
    """A run that ends by time: the time moves on while a step runs, also when its group has left before it; the step still
    belongs to the run."""
    p, d = make("recovery_nuclei", tmp_path)
    t = oracle.run(p, d)["trace"]["t"]
    for k in (20, 21, 33, 50):
        p, _ = make("recovery_nuclei", tmp_path, tmax=repr(float(0.5 * (t[k - 1] + t[k]))))
        ref = oracle.run(p, d)
        assert len(ref["trace"]) == k + 1
        for lim in ({"host_polls": 1}, {"host_polls": 1, "slots": 500}, {}):
            tr, labels, counts, _ = run(p, d, **lim)
            assert_same(tr, labels, *counts, ref)


@pytest.mark.parametrize("kind", ["requests", "depleted"])
def test_more_than_the_mailbox_holds(gpu, tmp_path, kind):
    """A step that asks for more than 16,384 weights, or in which more deformed grains than that lose their last cell, is finished
    after its launch."""
    if kind == "requests":
        n, par = 80, {"mobility_model": 2, "RH_exponent": "1.0"}
        d = sg.generate_domain(n, n, n, 20000, 16000, seed=9, device=0)
    else:
        # cells of one front speed finish together, in grains of one or two cells
        n, par = 64, {"mobility_model": 2}
        d = sg.generate_domain(n, n, n, 250000, 6000, seed=9, device=0, rho_sigma=0.0)
    p = sg.read_uds(sg.UdsSpec(nx=n, ny=n, nz=n, border_policy=1, **par).write(tmp_path / "p.uds"))
    out = [run(p, d, use_graph=g) for g in (1, 0)]
    tr = out[0][0]
    assert out[0][3] < 5 * len(tr)
    if kind == "requests":
        assert max(s.p_misses for s in tr) > 16384
        assert_same(*out[0][:2], *out[0][2], oracle.run(p, d))
    else:
        assert max(s.n_full for s in tr) > 40000
    assert np.array_equal(as_array(tr), as_array(out[1][0])) and np.array_equal(out[0][1], out[1][1])
    assert all(np.array_equal(a, b) for a, b in zip(out[0][2], out[1][2]))


@pytest.mark.parametrize("polls", [1, 4096])
def test_more_than_the_mailbox_holds_in_a_batch(gpu, tmp_path, polls):
    """The others' pending answers move with those of the domain that overflows."""
    n = 80
    big = sg.read_uds(sg.UdsSpec(nx=n, ny=n, nz=n, border_policy=1, mobility_model=2, RH_exponent="1.0").write(tmp_path / "p.uds"))
    cases = [(big, sg.generate_domain(n, n, n, 20000, 16000, seed=s, device=0)) for s in (9, 10)]
    for name in ("odd_periodic", "heating_rh", "recovery_nuclei"):
        cases.insert(1, make(name, tmp_path))
    with sg.Batch([p for p, _ in cases]) as b:
        set_limits(b, host_polls=polls)
        for i, (_, d) in enumerate(cases):
            b.load_domain(i, d)
        b.place_nuclei()
        b.run_until()
        assert max(s.p_misses for s in b.trace(0)) > 16384
        for i, (p, d) in enumerate(cases):
            assert_same(b.trace(i), b.labels(i), *b.grain_counts(i), oracle.run(p, d))
