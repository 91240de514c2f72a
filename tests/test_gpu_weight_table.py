"""The device weight table at the edges of its tiles and of its FP32 classification, against the host.

Rows and columns end inside and at a block's 8 x 256; orientation pairs sit on both sides of every threshold
(15 degrees, 30 and 50 degrees, 10 degrees from 40 deg <111>, the sigmoid's saturation) at 1e-7 to 1e-3 rad,
where FP32 alone could not tell; quaternions that are not of unit length go through FP64.
"""
import numpy as np
import pytest

import score_gb300 as sg
from score_gb300 import _abi
from test_zz_no_alloc import ATOL, _axis_angle, _qmul, _unit, device_table, host_table, orientations, rh_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrxg,ndefg", [(1, 1), (7, 255), (8, 256), (9, 257), (3, 2049), (700, 33)])
@pytest.mark.parametrize("model", [1, 2])
def test_table_sizes(gpu, nrxg, ndefg, model):
    p = sg.default_params() if model == 1 else rh_params()
    qr, qd = orientations(nrxg + ndefg, nrxg, ndefg)
    tab, pmax = device_table(_abi.load(), p, qr, qd)
    ref = host_table(p, qr, qd)
    assert np.abs(tab - ref).max() <= ATOL
    assert abs(pmax - ref.max()) <= ATOL
    const = (ref == -1.0) | (ref == 0.0) | (ref == 1.0)
    assert np.array_equal(tab[const], ref[const])


def threshold_pairs(rng):
    """Rotations q d with the misorientation on both sides of the thresholds; d uniform."""
    off = np.concatenate([s * 10.0 ** np.arange(-7, -2.5, 0.5) for s in (-1.0, 1.0)])
    rot = []
    for deg in (15.0, 30.0, 50.0):
        for axis in ([0, 0, 1], [1, 1, 1], [1, 2, 3]):
            rot.append(_axis_angle(np.tile(axis, (len(off), 1)), deg + np.degrees(off)))
    # 40 deg <111> followed by a rotation of 10 degrees and a little
    dev = _axis_angle(rng.normal(size=(len(off), 3)), 10.0 + np.degrees(off))
    rot.append(_qmul(np.broadcast_to(_axis_angle(np.ones((1, 3)), np.array([40.0])), dev.shape), dev))
    for cut in (1.0, 2.0):  # around the angle from which the sigmoid is 1 (exponents 4 and 9)
        sat = 15.0 * (60.0 / 5.0) ** (1.0 / (4.0 * cut))
        rot.append(_axis_angle(np.tile([1, 0, 0], (len(off), 1)), sat + np.degrees(off)))
    rot = np.concatenate(rot)
    d = _unit(rng.normal(size=(16, 4)))
    return np.ascontiguousarray(_unit(np.concatenate([_qmul(np.broadcast_to(x, rot.shape), rot) for x in d]))), np.ascontiguousarray(d)


def families(p, q):
    """The 24 equivalents of conj(q) p in 64 bits, (..., 6, 4)."""
    a, b, c, d = np.moveaxis(_qmul(q * np.array([1.0, -1.0, -1.0, -1.0]), p), -1, 0)
    f = 1.0 / np.sqrt(2.0)
    return np.stack([np.stack([(a + b) * f, (a - b) * f, (c + d) * f, (c - d) * f], -1),
                     np.stack([(a + c) * f, (a - c) * f, (b + d) * f, (b - d) * f], -1),
                     np.stack([(a + d) * f, (a - d) * f, (b + c) * f, (b - c) * f], -1),
                     np.stack([a + b + c + d, a + b - c - d, a - b + c - d, a - b - c + d], -1) * 0.5,
                     np.stack([a + b + c - d, a + b - c + d, a - b + c + d, a - b - c - d], -1) * 0.5,
                     np.stack([a, b, c, d], -1)], -2)


def sebald_gottstein(qr, qd):
    """The weight with both disorientations always taken, as the table takes them.  The host skips the second
    where the first angle is more than 10 degrees from 40 (a bound that holds for unit quaternions only)."""
    def angle(om):
        return np.where(om < 1.0 - 5.0e-16, 2.0 * np.arccos(np.minimum(om, 1.0)), 0.0)
    c = families(qr[:, None, :], qd[None, :, :])
    best = np.abs(c).max(-1)
    mi = best.argmax(-1)
    theta = angle(best.max(-1))
    dis = -np.sort(-np.abs(np.take_along_axis(c, mi[..., None, None], -2)[..., 0, :]), -1)
    h = np.pi / 9.0
    m40 = np.array([np.cos(h)] + [np.sin(h) / np.sqrt(3.0)] * 3)
    dev = angle(np.abs(families(dis, m40)).max((-1, -2)))
    ten = np.radians(10.0)
    w = np.where(dev < ten, np.cos(0.5 * np.pi * dev / ten) ** 2, 0.0)
    return np.where(theta <= np.radians(15.0), -1.0, w)


@pytest.mark.parametrize("model", [1, 2])
@pytest.mark.parametrize("length", [1.0, 1.02])
def test_table_at_thresholds(gpu, model, length):
    p = sg.default_params() if model == 1 else rh_params()
    qr, qd = threshold_pairs(np.random.default_rng(5))
    qr = qr * length
    tab, _ = device_table(_abi.load(), p, qr, qd)
    ref = host_table(p, qr, qd) if model == 2 or length == 1.0 else sebald_gottstein(qr, qd)
    assert np.abs(tab - ref).max() <= ATOL
