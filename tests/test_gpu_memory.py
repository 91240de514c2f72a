"""Device memory of a loaded domain and of post-processing: no list or workspace beyond what the domain's arrays take."""
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
