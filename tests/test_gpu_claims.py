"""Separate claim and resolve kernels of a batch (four lanes a full cell) against the oracle.

Domains of one step share the launches, so the sizes put a domain's end inside a warp's eight cells, leave domains
without full cells between others, and give both lists' cells, faces included, to one tile.  FP64: the
oracle's bits; the separate kernels of a single domain are covered by the other growth tests.
"""
import pytest

import oracle
import score_gb300 as sg
from test_gpu_fused import make
from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("names", [["one_nucleus", "odd_periodic", "one_tile"], ["thin", "many_full", "one_nucleus", "thin"]])
def test_batch_by_separate_kernels(gpu, tmp_path, names):
    cases = {n: make(n, tmp_path) for n in set(names)}
    refs = {n: oracle.run(p, d) for n, (p, d) in cases.items()}
    with sg.Batch([cases[n][0] for n in names]) as b:
        b.set_tune(use_graph=0)
        for i, n in enumerate(names):
            b.load_domain(i, cases[n][1])
        b.place_nuclei()
        steps = b.run_until()
        assert b.timing().kernel_launches >= 5 * steps
        for i, n in enumerate(names):
            assert_same(b.trace(i), b.labels(i), *b.grain_counts(i), refs[n])


def test_batch_changes_paths_on_the_way(gpu, tmp_path):
    """A batch whose fronts outgrow the launch's blocks goes on with the separate kernels, and back."""
    names = ["odd_periodic", "one_nucleus", "many_full", "thin"]
    cases = [make(n, tmp_path) for n in names]
    with sg.Batch([p for p, _ in cases]) as b:
        for i, (_, d) in enumerate(cases):
            b.load_domain(i, d)
        b.place_nuclei()
        traces = [[] for _ in names]
        for k in range(6):
            b.set_tune(use_graph=k % 2)
            b.run_until(max_steps=5)
            for i in range(len(names)):
                traces[i] += b.trace(i)
        b.set_tune(use_graph=1)
        b.run_until()
        for i, (p, d) in enumerate(cases):
            assert_same(traces[i] + b.trace(i), b.labels(i), *b.grain_counts(i), oracle.run(p, d))
