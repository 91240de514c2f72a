"""Percolation at boxes whose rows and columns end inside a packed word, on patterns set by the nuclei alone (a placed
nucleus is a 1-cell): nothing, one cell, a checkerboard, random fillings, everything, a comb whose teeth join late."""
import numpy as np
import pytest

import oracle
import score_gb300 as sg

pytestmark = pytest.mark.gpu


def pattern(kind, shape, rng):
    nz, ny, nx = shape
    z, y, x = np.indices(shape)
    if kind == "none":
        return np.zeros(shape, bool)
    if kind == "one":
        m = np.zeros(shape, bool)
        m[nz - 1, ny - 1, nx - 1] = True
        return m
    if kind == "checkerboard":
        return (x + y + z) % 2 == 1
    if kind == "all":
        return np.ones(shape, bool)
    if kind == "comb":
        return (x % 2 == 0) | (z == nz - 1)
    return rng.random(shape) < (0.31 if kind == "random" else 0.6)


@pytest.mark.parametrize("box", [(3, 3, 3), (5, 33, 4), (33, 32, 31), (64, 65, 3), (40, 7, 70), (31, 100, 9)])
@pytest.mark.parametrize("kind", ["none", "one", "checkerboard", "all", "comb", "random", "dense"])
def test_clusters(gpu, tmp_path, box, kind):
    nx, ny, nz = box
    m = pattern(kind, (nz, ny, nx), np.random.default_rng(nx + ny + nz))
    sites = np.flatnonzero(m.ravel()).astype(np.uint32)
    late = sites.size == 0  # a nucleus that is not due keeps the pool from being empty
    s = np.array([0], dtype=np.uint32) if late else sites
    p = sg.read_uds(sg.UdsSpec(nx=nx, ny=ny, nz=nz, border_policy=1).write(tmp_path / "p.uds"))
    d = sg.Domain(nx, ny, nz, np.zeros((nz, ny, nx), dtype=np.uint32), np.array([[1.0, 0.0, 0.0, 0.0]]), np.array([1e15]),
                  np.tile([0.0, 1.0, 0.0, 0.0], (s.size, 1)), s, np.full(s.size, 1e9 if late else 0.0))
    with sg.GrowthMachine(p) as gm:
        gm.load_domain(d)
        assert gm.place_nuclei() == sites.size
        for connected in (False, True):
            got = gm.percolation(connected=connected, labels=True)
            want = oracle.percolation(m.astype(np.uint8), nx, ny, nz, reference_scan=not connected)
            assert np.array_equal(got["labels"].ravel(), want["labels"])
            for f in ("n_clusters", "largest", "percolates", "spans"):
                assert got[f] == want[f], f
            assert np.array_equal(got["sizes"], want["sizes"])
        assert np.array_equal(gm.labels().ravel() != 0, m.ravel())  # the analysis leaves the state alone
