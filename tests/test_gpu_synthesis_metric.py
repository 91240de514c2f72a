"""The device label fill where the metric's scale leaves the range of FP32 squares, or one axis counts for next to nothing beside
another: the host's labels."""
import numpy as np
import pytest

import score_gb300 as sg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("aspect", [(1e22, 1e22, 1e22), (1e-25, 1e-25, 1e-25), (1e30, 1.0, 1.0), (1.0, 1e-30, 1.0), (1e20, 1e-20, 1.0),
                                    (3e18, 1e18, 2e18), (1e5, 1.0, 1e-5)])
@pytest.mark.parametrize("box,grains", [((20, 22, 18), 60), ((33, 9, 14), 700)])
def test_labels_equal_host(gpu, aspect, box, grains):
    host = sg.generate_domain(*box, grains, 5, seed=3, aspect=aspect)
    dev = sg.generate_domain(*box, grains, 5, seed=3, aspect=aspect, device=0)
    assert np.array_equal(dev.grid, host.grid)
