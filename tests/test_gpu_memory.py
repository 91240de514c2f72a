"""Device memory of a loaded domain and of post-processing: no list or workspace beyond what the domain's arrays take."""
import numpy as np
import pytest

import score_gb300 as sg

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
