"""The loaded grid's cells per deformed grain, at boxes whose edges end inside a brick or a warp's 8 x 2 x 2 box,
with one grain, grains of single cells and rows that change grain at every cell."""
import numpy as np
import pytest

import score_gb300 as sg
from score_gb300 import _abi

pytestmark = pytest.mark.gpu


def grid_of(kind, shape, rng):
    nz, ny, nx = shape
    if kind == "one":
        return np.zeros(shape, dtype=np.uint32), 1
    if kind == "single_cells":
        return np.arange(nx * ny * nz, dtype=np.uint32).reshape(shape), nx * ny * nz
    if kind == "stripes":
        return np.broadcast_to((np.arange(nx) % 3).astype(np.uint32), shape).copy(), 3
    return rng.integers(0, 7, size=shape).astype(np.uint32), 7


@pytest.mark.parametrize("box", [(3, 3, 3), (7, 5, 3), (8, 2 * 8, 4), (9, 17, 33), (65, 31, 6)])
@pytest.mark.parametrize("kind", ["one", "single_cells", "stripes", "random"])
def test_cells_per_grain(gpu, tmp_path, box, kind):
    nx, ny, nz = box
    rng = np.random.default_rng(nx * ny * nz)
    grid, ng = grid_of(kind, (nz, ny, nx), rng)
    quat = np.tile([1.0, 0.0, 0.0, 0.0], (ng, 1))
    p = sg.read_uds(sg.UdsSpec(nx=nx, ny=ny, nz=nz, border_policy=1).write(tmp_path / "p.uds"))
    d = sg.Domain(nx, ny, nz, grid, quat, np.full(ng, 1e15), np.array([[0.0, 1.0, 0.0, 0.0]]), np.array([nx * ny * nz // 2], dtype=np.uint32),
                  np.zeros(1))
    with sg.GrowthMachine(p) as gm:
        for _ in range(2):  # the second load counts into the same words
            gm.load_domain(d)
            rx, deformed = gm.grain_counts()
            assert np.array_equal(deformed, np.bincount(grid.ravel(), minlength=ng)) and not rx.any()
            assert np.array_equal(gm.labels(), grid)
        bad = grid.copy()
        bad[nz - 1, ny - 1, nx - 1] = ng
        with pytest.raises(sg.ScoreError) as e:
            gm.load_domain(sg.Domain(nx, ny, nz, bad, quat, d.defg_rho0, d.rxg_quat, d.rxg_site, d.rxg_tincub))
        assert e.value.status == _abi.ERR_ARG
