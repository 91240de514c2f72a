"""Weights of quaternions that are not quite of unit length (rounded to a few digits in an input file): FP32 may settle a pair only
where the formula in 64 bits gives the same constant for the lengths as they are."""
import numpy as np
import pytest

import score_gb300 as sg
from score_gb300 import _abi
from test_gpu_weight_table import sebald_gottstein, threshold_pairs
from test_zz_no_alloc import ATOL, _axis_angle, _qmul, _unit, device_table, host_table

pytestmark = pytest.mark.gpu

LENGTHS = [1.0 + s * d for d in (4e-4, 2e-4, 5e-5, 1e-5, 4e-6, 2e-6, 1e-6) for s in (1.0, -1.0)]


def pairs():
    """Both sides of every threshold, and rotations about <111> within 0.3 degrees of 30 and 50 degrees, where the length of the
    quaternion decides between the two sides."""
    rng = np.random.default_rng(8)
    qr, qd = threshold_pairs(rng)
    deg = np.concatenate([c + rng.uniform(-0.3, 0.3, 64) for c in (30.0, 50.0)])
    axis = np.ones((len(deg), 3)) + rng.normal(scale=1e-3, size=(len(deg), 3))
    near = _unit(_qmul(np.broadcast_to(qd[0], (len(deg), 4)), _axis_angle(axis, deg)))
    return np.concatenate([qr, near]), qd


@pytest.mark.parametrize("length", LENGTHS)
def test_table(gpu, length):
    qr, qd = pairs()
    qr = np.ascontiguousarray(qr * length)
    tab, pmax = device_table(_abi.load(), sg.default_params(), qr, qd)
    ref = sebald_gottstein(qr, qd)
    assert np.abs(tab - ref).max() <= ATOL and abs(pmax - ref.max()) <= ATOL


@pytest.mark.parametrize("length", [1.0004, 0.9998, 1.00002])
def test_growth_takes_the_hosts_weights(gpu, tmp_path, length):
    """A run that settles its pairs itself against one that is given the host's table."""
    qr, qd = pairs()
    p = sg.read_uds(sg.UdsSpec(nx=64, ny=64, nz=64, border_policy=1).write(tmp_path / "p.uds"))
    d = sg.generate_domain(64, 64, 64, len(qd), 400, seed=12)
    pick = np.random.default_rng(1).permutation(len(qr))[:400]
    pick[:128] = np.arange(len(qr) - 128, len(qr))
    d.rxg_quat[:] = qr[pick] * length
    d.defg_quat[:] = qd
    out = []
    for table in (None, host_table(p, d.rxg_quat, d.defg_quat)):
        with sg.GrowthMachine(p) as gm:
            gm.load_domain(d, table)
            gm.place_nuclei()
            tr = gm.run_until()
            out.append((np.array([(s.t, s.Xcells, s.Sv, s.n_new) for s in tr]), gm.labels()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
