"""Two contexts on two host threads whose launches each want the whole GPU take turns of a launch: neither is left with a step
or two a launch while the other runs, and the results are those of a context alone."""
import threading

import numpy as np
import pytest

import score_gb300 as sg

pytestmark = pytest.mark.gpu


def test_contexts_take_turns(gpu, tmp_path):
    p = sg.read_uds(sg.UdsSpec(nx=256, ny=256, nz=256).write(tmp_path / "p.uds"))
    doms = [sg.generate_domain(256, 256, 256, 2000, 5000, seed=s, device=0) for s in (1, 2)]
    runs = 3
    out = [None, None]
    gate = threading.Barrier(2)

    def work(k, together):
        with sg.GrowthMachine(p) as gm:
            gm.load_domain(doms[k])
            got = []
            for _ in range(runs):
                gm.restart()
                gm.place_nuclei()
                n0 = gm.timing().kernel_launches
                if together:
                    gate.wait(60)
                tr = gm.run_until()
                got.append((gm.timing().kernel_launches - n0, len(tr), tr[-1].t, gm.labels()))
            out[k] = got

    for k in range(2):
        work(k, False)
    alone = list(out)
    th = [threading.Thread(target=work, args=(k, True)) for k in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join(120)
    for k in range(2):
        for (_, steps, t, labels), (_, steps0, t0, labels0) in zip(out[k], alone[k]):
            assert steps == steps0 and t == t0 and np.array_equal(labels, labels0)
    # 12 launches of 30 steps alone; as many and one or two more where every launch has its turn, 23 for the one whose turn has
    # passed when it comes out of the queue
    worst = sorted(max(out[0][r][0] - alone[0][r][0], out[1][r][0] - alone[1][r][0]) for r in range(runs))
    assert worst[runs // 2] <= 5, worst
