"""The device label fill at the edges of its buckets, bit for bit against the host generator: one seed, few seeds (every
bucket is a neighbour, by either image), as many seeds as cells, flat boxes, flattened metrics, and more seeds around
a bucket than shared memory holds."""
import numpy as np
import pytest

import score_gb300 as sg

pytestmark = pytest.mark.gpu

CASES = [((5, 7, 3), 1, {}), ((33, 17, 9), 2, {}), ((40, 40, 40), 9, {}), ((64, 48, 56), 27, {}), ((61, 83, 47), 200, {}),
         ((96, 96, 3), 300, {}), ((1, 1, 300), 40, {}), ((16, 16, 16), 4096, {}), ((30, 30, 30), 20000, {}),
         ((128, 90, 70), 150, {"aspect": (1.0, 4.0, 8.0)}), ((70, 130, 50), 1000, {"aspect": (8.0, 1.0, 2.5)}),
         ((200, 8, 8), 64, {"aspect": (0.25, 1.0, 1.0)})]


@pytest.mark.parametrize("box,grains,kw", CASES)
@pytest.mark.parametrize("seed", [1, 2])
def test_labels_equal_host(gpu, box, grains, kw, seed):
    nuclei = min(5, box[0] * box[1] * box[2])
    host = sg.generate_domain(*box, grains, nuclei, seed=seed, **kw)
    dev = sg.generate_domain(*box, grains, nuclei, seed=seed, device=0, **kw)
    assert np.array_equal(dev.grid, host.grid)
    assert np.array_equal(dev.rxg_site, host.rxg_site) and np.array_equal(dev.defg_quat, host.defg_quat)
